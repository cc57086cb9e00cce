// mps_ops.cu — the per-particle operators of the PolyMPS step on sm_103a.
//
// One thread per particle i, or 8 or 4 lanes in small systems (lanesFor).  Sweeps at the
// post-prediction positions walk the ELL neighbour row of i (built once per position epoch
// through the stale bucket list, in the reference's scan order); the start-of-step viscosity and
// the post-correction shifting read the start-of-step skin list and its filter.  With the skin
// list off both walk the 27 buckets, as the dummy velocities do.
// Membership (the reference's own radius and mirror-side tests) is decided first, from the FP32
// copies outside their rounding band and in exact FP64 inside it (see mps_common.cuh); the FP64
// sums then run over the members only.
#include "mps_df.cuh"
#include "mps_internal.h"
#include "mps_lanes.cuh"

#define BLK 128

// ------------------------------------------------------------------ viscosity
// MpsViscosity::calcViscosity, src/MpsViscosity.cpp:20-100 (Newtonian: MEU and RHO are
// uniform, src/MpsInputOutput.cpp:833-838, so the harmonic mean is hoisted).  Staged scan
// at the start-of-step positions; FP32 prefilter, exact FP64 radius/side tests.
// The kinematic factors of a wall and of a fluid neighbour, (2 mu)/rho and
// (2 mu mu / (mu + mu))/rho (src/MpsViscosity.cpp:55-62), are run constants (Dev).
struct ViscSum {
    dvec4 vi;
    double ax, ay, az;
    __device__ __forceinline__ void add(const Dev& d, dvec4 pi, int j) {
        const MpsParams& P = d.P;
        const PairG q = pairSum(d.pos[j], pi);
        double wL, wd;
        weightR(q.d2, P.reL, P.weightType, wL, wd);
        const double f = wL * ((d.type[j] == P.wall) ? d.neuWall64 : d.neuFluid64);
        const dvec4 vj = d.vel[j];
        ax += (vj.x - vi.x) * f; ay += (vj.y - vi.y) * f; az += (vj.z - vi.z) * f;
    }
};
struct OpViscosity {
    struct State { ViscSum v; SideCtx sc; dvec4 pi; };
    __device__ float hi(const Dev& d) const { return d.bandHiL; }
    __device__ bool active(const Dev&, const State&) const { return true; }
    __device__ void begin(const Dev& d, int i, State& st) const {
        st.v = {d.vel[i], 0.0, 0.0, 0.0};
        st.pi = d.pos[i];
        st.sc = sideCtx(d, i, st.pi);
    }
    __device__ void visit(const Dev& d, int i, State& st, int j, dvec4 pj, PairG q) const {
        if (!(q.d2 < d.P.reL2) || !sideOK(st.sc, pj, q.d2)) return;
        st.v.add(d, st.pi, j);
    }
    __device__ void end(const Dev& d, int i, State& st) const {
        double c = d.P.coeffViscMultiphase;
        d.acc[i] = make_dvec4(c * st.v.ax, c * st.v.ay, c * st.v.az, 0.0);
    }
};
void launchViscosity(const Dev& d, cudaStream_t s) {
    launchScan(d, OpViscosity(), s);
}
// The same sweep over the start-of-step skin list (built just before from the same FP32
// copies), L lanes per particle.  The list holds about 56 entries a row for the 32 inside
// reL: the FP32 copies decide them first, and the FP64 sums (bound by the FP64 pipe, about 20
// operations an entry) walk only those inside: 2,252 -> 1,066 us at 864k particles, 114 -> 22
// at 6.9k.  A row that overflowed the list capacity
// (count K + 1) scans the buckets with its first lane.
template <int L>
__global__ void __launch_bounds__(128) k_visc_list(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const dvec4 pi = d.pos[i];
    const float4 fi = d.posf[i];
    ViscSum v = {d.vel[i], 0.0, 0.0, 0.0};
    const int c = d.nbrCount[i];
    if (c <= d.K) {
        const int* row = d.nbr + i;
        const SideF sd = sideF(d, i, pi);
        const Mask m = rowMask<L>(d, row, l, c, [&](int j, float4 hj) {
            const float d2f = dist2f(hj, fi);
            return insideF(d, d2f, d.bandLoL, d.bandHiL, d.P.reL2, i, j) && sideOKF(d, sd, hj, d2f, i, j);
        });
        forBits(row, d.N0, m, [&](int j, int) { v.add(d, pi, j); });
    } else if (l == 0) {
        const SideCtx sc = sideCtx(d, i, pi);
        forCellsNear(d, pi, fi, d.bandHiL, [&](int j, dvec4 pj, PairG q) {
            if (j != i && q.d2 < d.P.reL2 && sideOK(sc, pj, q.d2)) v.add(d, pi, j);
        });
    }
    const double ax = laneSum<L>(v.ax), ay = laneSum<L>(v.ay), az = laneSum<L>(v.az);
    const double cv = d.P.coeffViscMultiphase;
    if (l == 0) d.acc[i] = make_dvec4(cv * ax, cv * ay, cv * az, 0.0);
}
void launchViscosityList(const Dev& d, cudaStream_t s) {
#define LAUNCH(L) k_visc_list<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// List of the current positions filtered from the skin list: the set, order and (WEIGHTS, the
// FP64 tier) per-entry weights of k_build_list, L lanes per particle.  Membership (d^2 <
// reMax^2) comes from the FP32 copies outside their rounding band; the weights, the FP64
// part, are then formed over the members only (864k particles: 1,699 -> 992 us; decided and
// formed entry by entry, every warp issued the weights for 56 entries instead of 33).  A
// particle whose scan window changed or whose skin row overflowed, or every particle once the
// skin list went stale, is left to k_rescan: a few particles cross a bucket face in every
// step, and scanned in place one lane's walk of 27 buckets was the time of the whole kernel
// (108k particles with weights 226 us, without them 98; now 130 + 14 and 32 + 13 us).
template <bool WEIGHTS, int L>
__global__ void __launch_bounds__(128) k_filter_nbr(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const dvec4 pi = d.pos[i];
    const float4 fi = d.posf[i];
    const size_t N0 = d.N0;
    const int c = d.skinCnt[i];
    int cnt = 0;
    if (!*(volatile int*)d.skinFlag && c <= d.K && d.skinCell[i] == cellKeyOf(d, pi, fi)) {
        const int* row = d.skinNbr + i;
        // without weights one lane appends as it decides: 393 us at 2.8M particles against
        // 672 with the second walk of the row (124 / 205 us at 864k)
        const bool direct = !WEIGHTS && L == 1;
        const Mask m = rowMask<L>(d, row, l, c, [&](int j, float4 hj) {
            const bool in = insideF(d, dist2f(hj, fi), d.bandLo, d.bandHi, d.reMax2, i, j);
            if (direct && in) d.nbr[(size_t)cnt++ * N0 + i] = j;
            return in && !direct;
        });
        const Mask all = laneOr<L>(m);
        if (!direct) cnt = maskCount(all);
        if (l == 0) d.nbrCount[i] = cnt;
        forBits(row, N0, m, [&](int j, int k) {
            const size_t e = (size_t)maskRank(all, k) * N0 + i;
            d.nbr[e] = j;
            if (WEIGHTS) storeWeights(d, e, pairSum(d.pos[j], pi).d2);
        });
    } else if (l == 0) {
        d.nearList[atomicAdd(d.rescan, 1)] = i;   // the near-wall list is written later (masks)
    }
    warpCount(d.counters, l == 0 ? (unsigned)cnt : 0u);
}
// The particles the filter left: the 27-bucket scan of k_build_list by one warp each.  The
// window's nine rows of three buckets are ranges of the bucket order of about 28 particles, one
// pass of the warp's lanes each; their bounds are loaded by nine lanes at once.
template <bool WEIGHTS>
__global__ void __launch_bounds__(128) k_rescan(Dev d) {
    const int lane = threadIdx.x & 31;
    const int n = *(volatile int*)d.rescan;
    const MpsParams& P = d.P;
    const size_t N0 = d.N0;
    for (int w = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += (int)(gridDim.x * blockDim.x) >> 5) {
        const int i = d.nearList[w];
        const dvec4 pi = d.pos[i];
        const float4 fi = d.posf[i];
        int ix, iy, iz;
        bucketCoordsHi(d, pi, fi, ix, iy, iz);
        int a = 0, b = 0;
        if (lane < (d.dz3 ? 9 : 3)) {
            const long long jb = (long long)((iz - 1) * d.dz3 + lane / 3) * P.numBucketsXY +
                                 (long long)(iy - 1 + lane % 3) * P.numBucketsX + ix;
            const long long lo = jb - 1 > 0 ? jb - 1 : 0, hi = jb + 1 < d.nB - 1 ? jb + 1 : d.nB - 1;
            if (lo <= hi) { a = d.cellStart[lo]; b = d.cellStart[hi + 1]; }
        }
        float4 f[9];   // the first pass over every range, loaded at once
#pragma unroll
        for (int r = 0; r < 9; r++) {
            const int s0 = __shfl_sync(0xffffffffu, a, r), s1 = __shfl_sync(0xffffffffu, b, r);
            if (s0 + lane < s1) f[r] = __ldg(&d.posf[__ldg(d.cellSorted + s0 + lane)]);
        }
        int cnt = 0;
#pragma unroll
        for (int r = 0; r < 9; r++) {
            const int s0 = __shfl_sync(0xffffffffu, a, r), s1 = __shfl_sync(0xffffffffu, b, r);
            for (int t = s0; t < s1; t += 32) {
                const int s = t + lane;
                int j = i;
                bool in = false;
                if (s < s1) {
                    j = __ldg(d.cellSorted + s);
                    const float d2f = dist2f(t == s0 ? f[r] : __ldg(&d.posf[j]), fi);
                    if (!(d2f > d.bandHi)) {
                        in = j != i && insideF(d, d2f, d.bandLo, d.bandHi, d.reMax2, i, j);
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, in);
                const int k = cnt + __popc(m & ((1u << lane) - 1u));
                if (in && k < d.K) d.nbr[(size_t)k * N0 + i] = j;
                cnt += __popc(m);
            }
        }
        if (WEIGHTS) {
            __syncwarp();
            for (int k = lane; k < cnt && k < d.K; k += 32) {
                const size_t e = (size_t)k * N0 + i;
                storeWeights(d, e, pairSum(d.pos[d.nbr[e]], pi).d2);
            }
        }
        if (lane == 0) {
            if (cnt > d.K) { setErr(d, MPSE_CAPACITY); cnt = d.K; }
            d.nbrCount[i] = cnt;
            if (cnt) atomicAdd(d.counters, (unsigned long long)cnt);
        }
    }
}
void launchNeighborFilter(const Dev& d, cudaStream_t s, bool weights, bool cells) {
    if (cells) {
        launchPosf(d, s);
        launchSkinCheck(d, s, true);
    } else {
        launchPosfCheck(d, s);
    }
#define LAUNCH(L)                                                                        \
    if (weights) k_filter_nbr<true, L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d);        \
    else k_filter_nbr<false, L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
    // the list's length is on the device: enough warps to fill the chip, at most one each
    const int grid = gridFor(d.N0, 4) < 1216 ? gridFor(d.N0, 4) : 1216;
    if (weights) k_rescan<true><<<grid, 128, 0, s>>>(d);
    else k_rescan<false><<<grid, 128, 0, s>>>(d);
}

// MpsParticle::addGravity, src/MpsParticle.cpp:111-130
__global__ void k_add_gravity(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    dvec4 a = d.acc[i];
    a.x += d.P.gravity[0]; a.y += d.P.gravity[1]; a.z += d.P.gravity[2];
    d.acc[i] = a;
    d.accStar[i] = a;
}
void launchAddGravity(const Dev& d, cudaStream_t s) { k_add_gravity<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }

// MpsParticleVelPos::predictionVelocityPosition, src/MpsParticleVelPos.cpp:20-50, with the
// acceleration a of particle i
__device__ __forceinline__ void predictParticle(const Dev& d, int i, dvec4 a) {
    const MpsParams& P = d.P;
    if (d.type[i] == P.fluid) {
        dvec4 v = d.vel[i], x = d.pos[i];
        v.x += a.x * P.timeStep; v.y += a.y * P.timeStep; v.z += a.z * P.timeStep;
        x.x += v.x * P.timeStep; x.y += v.y * P.timeStep; x.z += v.z * P.timeStep;
        d.vel[i] = v; d.pos[i] = x;
    }
    dvec4 z = make_dvec4(0, 0, 0, 0);
    d.acc[i] = z; d.dvel[i] = z; d.npcd[i] = z;
    d.nNeighWall[i] = 0;
    d.nearWall[i] = 0;
    double big = 10e8 * P.partDist;
    d.riw2[i] = big;
    if (P.wallType == 1) d.mirror[i] = make_dvec4(big, big, big, 0.0);
}
__global__ void k_predict(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < liveN(d)) predictParticle(d, i, d.acc[i]);
}
void launchPredict(const Dev& d, cudaStream_t s) { k_predict<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }
// both operators in one pass (a step without the prediction's pressure gradient between them)
__global__ void k_gravity_predict(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    dvec4 a = d.acc[i];
    a.x += d.P.gravity[0]; a.y += d.P.gravity[1]; a.z += d.P.gravity[2];
    d.accStar[i] = a;
    predictParticle(d, i, a);
}
void launchGravityPredict(const Dev& d, cudaStream_t s) { k_gravity_predict<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }

// ------------------------------------------------------------------ out of domain
// MpsParticle::checkParticleOutDomain, src/MpsParticle.cpp:270-396.  A parallel pass flags
// fluid particles outside [min + bucket, max - bucket] by reference index; when any is
// flagged, a single thread replays the reference's serial swap-with-last loop on reference
// indices: the data of the last live index is copied onto the removed one (the arrays the
// reference copies) and the last index becomes a ghost, exactly as in the reference, on
// the storage slots of those indices.  Live storage is then kept contiguous: the ghost's
// slot trades places with the last live slot (all arrays, the index maps and the two
// entries of the step's bucket list, so the list keeps pointing at the same data).
__device__ __forceinline__ bool outside(const Dev& d, dvec4 p) {
    return p.x > d.oodHi[0] || p.x < d.oodLo[0] || p.y > d.oodHi[1] || p.y < d.oodLo[1] ||
           (d.dz3 && (p.z > d.oodHi[2] || p.z < d.oodLo[2]));
}
template <class T> __device__ __forceinline__ void mv(T* a, int i, int L) { a[i] = a[L]; }
template <class T> __device__ __forceinline__ void sw(T* a, int i, int j) { T t = a[i]; a[i] = a[j]; a[j] = t; }
// every per-particle array that lives across operators: a pure relocation of two slots
__device__ void swapSlots(const Dev& d, int a, int b) {
    for (dvec4* v : {d.pos, d.vel, d.acc, d.accStar, d.mirror, d.wallPos, d.polyNormal, d.normal, d.npcd, d.gradC,
                     d.forceWall, d.c1, d.c2, d.c3, d.dvel, d.shift})
        sw(v, a, b);
    for (double* v : {d.press, d.pressPPE, d.pressPPEprev, d.pressPPEprev2, d.pndi, d.pndki, d.pndski, d.pndSmall, d.npcd2, d.conc,
                      d.velDiv, d.diffTerm, d.pndWall, d.riw2, d.devDot, d.source, d.aux1, d.aux2})
        sw(v, a, b);
    for (int* v : {d.type, d.bc, d.numNeigh, d.nNeighWall, d.nearWall, d.cellOf}) sw(v, a, b);
    sw(d.posf, a, b);
    sw(d.posLo, a, b);
    int ra = d.orig[a], rb = d.orig[b];
    d.orig[a] = rb; d.orig[b] = ra;
    d.slotOf[ra] = b; d.slotOf[rb] = a;
    int pa = d.cellPos[a], pb = d.cellPos[b];
    if (pa >= 0) d.cellSorted[pa] = b;
    if (pb >= 0) d.cellSorted[pb] = a;
    d.cellPos[a] = pb; d.cellPos[b] = pa;
}
__device__ void outSerial(const Dev& d, int* flags) {
    const MpsParams& P = d.P;
    const int oldN = *d.nLive;
    int newN = oldN;
    int removed = 0;
    for (int r = 0; r < newN; r++) {
        if (!flags[r]) continue;
        const int L = newN - 1;
        const int i = d.slotOf[r], l = d.slotOf[L];
        if (i != l) {
            mv(d.type, i, l); mv(d.bc, i, l); mv(d.numNeigh, i, l); mv(d.press, i, l); mv(d.pndi, i, l);
            mv(d.pndki, i, l); mv(d.pndski, i, l); mv(d.pndSmall, i, l); mv(d.npcd2, i, l); mv(d.conc, i, l);
            mv(d.velDiv, i, l); mv(d.diffTerm, i, l); mv(d.nearWall, i, l); mv(d.nNeighWall, i, l);
            mv(d.pndWall, i, l); mv(d.devDot, i, l); mv(d.riw2, i, l);
            if (P.mpsType == 2 || P.mpsType == 3) { mv(d.pressPPE, i, l); mv(d.source, i, l); mv(d.pressPPEprev, i, l); mv(d.pressPPEprev2, i, l); }
            mv(d.acc, i, l); mv(d.accStar, i, l); mv(d.pos, i, l); mv(d.vel, i, l); mv(d.npcd, i, l);
            mv(d.gradC, i, l); mv(d.c1, i, l); mv(d.c2, i, l); mv(d.c3, i, l); mv(d.dvel, i, l);
            mv(d.wallPos, i, l); mv(d.mirror, i, l); mv(d.polyNormal, i, l); mv(d.forceWall, i, l);
        }
        d.type[l] = P.ghost; d.bc[l] = P.other; d.nearWall[l] = 0; d.riw2[l] = 10e8 * P.partDist;
        d.vel[l] = make_dvec4(0, 0, 0, 0);
        d.press[l] = 0.0;
        d.pos[l] = make_dvec4(P.domainMax[0] - P.partDist, P.domainMax[1] - P.partDist,
                              (P.dim == 2) ? 0.0 : P.domainMax[2] - P.partDist, 0.0);
        if (l != newN - 1) swapSlots(d, l, newN - 1);
        newN--;
        removed++;
    }
    *d.nLive = newN;
    if (removed) d.skinFlag[0] = 1;   // indices moved: the start-of-step list is stale
    for (int r = 0; r < oldN; r++) flags[r] = 0;
}
// flags (by reference index) and the counters (flagged particles, blocks done) are zero between
// calls: only flagged particles write theirs, the serial pass clears what it read, and the last
// block to finish, which runs it, clears the counters.  Every block adds one to the same word, so
// the grid is at most four blocks per SM that stride over the particles: at 864k particles, cold
// cache, 15.7 us against 20.1 with a block per 256 particles and 17.5 with eight blocks per SM.
#define OUT_BLOCKS 608
__global__ void k_out_of_domain(Dev d, int* flags, int* counter) {
    const int n = liveN(d);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const dvec4 p = d.pos[s];
        if (d.type[s] == d.P.fluid && outside(d, p)) {
            flags[d.orig[s]] = 1;
            atomicAdd(counter, 1);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (atomicAdd(counter + 1, 1) != (int)gridDim.x - 1) return;
    __threadfence();
    if (*(volatile int*)counter) outSerial(d, flags);
    counter[0] = 0;
    counter[1] = 0;
}
void launchOutOfDomain(const Dev& d, int* flags, int* counter, cudaStream_t s) {
    const int grid = gridFor(d.N0, 256) < OUT_BLOCKS ? gridFor(d.N0, 256) : OUT_BLOCKS;
    k_out_of_domain<<<grid, 256, 0, s>>>(d, flags, counter);
}

// ------------------------------------------------------------------ collision
// MpsParticleCollision::checkParticleCollisions (PC), src/MpsParticleCollision.cpp:22-119:
// velocity corrections computed from the pre-collision velocities, then applied.
__global__ void __launch_bounds__(BLK) k_collision(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    dvec4 dv = make_dvec4(0, 0, 0, 0);
    if (d.type[i] == P.fluid) {
        double mi = P.DNS_FL1;  // PTYPE == 1 for every Newtonian particle
        dvec4 pi = d.pos[i], vi = d.vel[i];
        const float4 fi = d.posf[i];
        const SideCtx sc = d.mirrorFar ? SideCtx{} : sideCtx(d, i, pi);   // {}: no side test
        forNbrsPosf(d, i, [&](int j, float4 fj) {
            // FP32 prefilter (the list's FP32 copies): most entries lie beyond the collision
            // distance; the exact FP64 test decides the others
            const float ex = fj.x - fi.x, ey = fj.y - fi.y, ez = fj.z - fi.z;
            if (ex * ex + ey * ey + ez * ez > d.bandHiColl) return;
            dvec4 pj = d.pos[j];
            PairG q = pairOf(pj, pi);
            if (q.d2 < P.distCollisionLimit2 && sideOK(sc, pj, q.d2)) {
                dvec4 vj = d.vel[j];
                double fDT = (vi.x - vj.x) * q.v0 + (vi.y - vj.y) * q.v1 + (vi.z - vj.z) * q.v2;
                if (fDT > 0.0) {
                    bool jf = d.type[j] == P.fluid;
                    double mj = jf ? P.DNS_FL1 : P.densityWall;
                    fDT *= P.restitutionCollision * mj / (mi + mj) / q.d2;
                    double f = jf ? 1.0 : 2.0;
                    dv.x -= f * q.v0 * fDT; dv.y -= f * q.v1 * fDT; dv.z -= f * q.v2 * fDT;
                }
            }
        });
    }
    d.dvel[i] = dv;
}
__global__ void k_collision_apply(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    if (d.type[i] == d.P.fluid) {
        dvec4 v = d.vel[i], dv = d.dvel[i];
        v.x += dv.x; v.y += dv.y; v.z += dv.z;
        d.vel[i] = v;
    }
    d.dvel[i] = make_dvec4(0, 0, 0, 0);
}
void launchCollisionApply(const Dev& d, cudaStream_t s) {
    k_collision_apply<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
}
void launchCollision(const Dev& d, cudaStream_t s) {
    k_collision<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    launchCollisionApply(d, s);
}

// MpsParticleCollision::checkDynamicParticleCollisions (DPC, collision type 1),
// src/MpsParticleCollision.cpp:120-292: list entries closer than l0 off the mirror side;
// approaching pairs exchange momentum with kappa (1 below l0/2, else chi =
// sqrt(W_ij / W(l0/2)), W = (1 - r/l0)^4 (4 r/l0 + 1)), separating pairs get the dynamic
// background-pressure repulsion; then v += dv, x += dv dt for fluid particles.
__global__ void __launch_bounds__(BLK) k_collision_dpc(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    dvec4 dv = make_dvec4(0, 0, 0, 0);
    const MpsParams& P = d.P;
    if (d.type[i] == P.fluid) {
        const double mi = P.DNS_FL1;   // PTYPE == 1 for every Newtonian particle
        const double Wij5 = 0.5 * 0.5 * 0.5 * 0.5 * 3.0;
        const double gMod = sqrt(P.gravity[0] * P.gravity[0] + P.gravity[1] * P.gravity[1] + P.gravity[2] * P.gravity[2]);
        const double l02 = P.partDist * P.partDist;
        const double pmax = 2.0 / 3.0 * P.DNS_FL1 * gMod * 0.2, pmin = P.DNS_FL1 * gMod * P.partDist;
        const dvec4 pi = d.pos[i], vi = d.vel[i];
        const double pri = d.press[i];
        SideCtx sc = sideCtx(d, i, pi);
        forNbrs(d, i, [&](int j) {
            dvec4 pj = d.pos[j];
            PairG q = pairOf(pj, pi);
            if (!(q.d2 < l02 && sideOK(sc, pj, q.d2))) return;
            const bool jf = d.type[j] == P.fluid;
            const double mj = jf ? P.DNS_FL1 : P.densityWall;
            const double dst = sqrt(q.d2);
            double Wij = 0.0;
            if (dst > P.epsilonZero) {
                double w1 = 1.0 - dst * P.invPartDist;
                double w2 = 4.0 * dst * P.invPartDist + 1.0;
                Wij = w1 * w1 * w1 * w1 * w2;
            }
            const double chi = sqrt(Wij / Wij5);
            const double kappa = (dst < 0.5 * P.partDist) ? 1.0 : chi;
            const dvec4 vj = d.vel[j];
            double fDT = (vi.x - vj.x) * q.v0 + (vi.y - vj.y) * q.v1 + (vi.z - vj.z) * q.v2;
            const double f2 = jf ? 1.0 : 2.0;
            double k;
            if (fDT > 0.0) {
                k = fDT * kappa * 2.0 * mj / (mi + mj) / q.d2;
            } else {
                double ptil = fmax(fmin(P.lambdaCollision * fabs(pri + d.press[j]), P.lambdaCollision * pmax), pmin);
                double pb = ptil * chi;
                k = P.timeStep / mi * chi * pb / q.d2;
            }
            dv.x -= f2 * q.v0 * k; dv.y -= f2 * q.v1 * k; dv.z -= f2 * q.v2 * k;
        });
    }
    d.dvel[i] = dv;
}
__global__ void k_collision_dpc_apply(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    if (d.type[i] == d.P.fluid) {
        dvec4 v = d.vel[i], x = d.pos[i], dv = d.dvel[i];
        const double dt = d.P.timeStep;
        v.x += dv.x; v.y += dv.y; v.z += dv.z;
        x.x += dv.x * dt; x.y += dv.y * dt; x.z += dv.z * dt;
        d.vel[i] = v;
        d.pos[i] = x;
    }
    d.dvel[i] = make_dvec4(0, 0, 0, 0);
}
void launchCollisionDPC(const Dev& d, cudaStream_t s) {
    k_collision_dpc<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    k_collision_dpc_apply<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
}

// ------------------------------------------------------------------ wall NPCD
// Wall-only sweeps run over the compacted list of fluid particles near the wall.
__device__ __forceinline__ int nearIndex(const Dev& d) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    return (t < *d.nearCount) ? d.nearList[t] : -1;
}
// MpsPndNeigh::calcWallNPCD, src/MpsPndNeigh.cpp:105-195
__global__ void __launch_bounds__(WALL_BLK) k_wall_npcd(Dev d) {
    __shared__ double sm[3][32];
    const MpsParams& P = d.P;
    forNearWall(d, [](int, int) {}, [&](int i, int g, int l) {
        const dvec4 mi = d.mirror[i];
        double dx = 0, dy = 0, dz = 0;
        forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorS[i], l, [&](int j, int) {
            const PairG m = pairSum(d.pos[j], mi);
            double wS, wd;
            weightR(m.d2, P.reS, P.weightType, wS, wd);
            dx += m.v0 * wS; dy += m.v1 * wS; dz += m.v2 * wS;
        });
        dx = laneSum<WALL_L>(dx); dy = laneSum<WALL_L>(dy); dz = laneSum<WALL_L>(dz);
        if (l == 0) { sm[0][g] = dx; sm[1][g] = dy; sm[2][g] = dz; }
    }, [&](int i, int g) {
        const dvec4 pi = d.pos[i], mi = d.mirror[i];
        const ReflG r = makeRefl(pi, mi, P.epsilonZero, true);
        double dx = sm[0][g], dy = sm[1][g], dz = sm[2][g];
        PairM s = pairMirror(pi, mi);
        if (s.dm2 < P.reS2) {
            double wS = wfun(sqrt(s.dm2), P.reS, P.weightType);
            dx += s.m0 * wS; dy += s.m1 * wS; dz += s.m2 * wS;
        }
        dvec4 n = d.npcd[i];
        n.x += r.R[0] * dx + r.R[1] * dy + r.R[2] * dz;
        n.y += r.R[3] * dx + r.R[4] * dy + r.R[5] * dz;
        n.z += r.R[6] * dx + r.R[7] * dy + r.R[8] * dz;
        d.npcd[i] = n;
    });
}
void launchWallNpcd(const Dev& d, cudaStream_t s) {
    if (d.P.wallType != 1) return;
    k_wall_npcd<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ velocity divergence
// MpsPressure::calcVelDivergence, src/MpsPressure.cpp:479-557: fluid particles over the reS
// entries off the mirror side; PND-weighted, or through the correction matrix.
__global__ void __launch_bounds__(BLK) k_vel_div(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    double div = 0.0;
    if (d.type[i] == P.fluid) {
        const double ni = d.pndi[i];
        const dvec4 pi = d.pos[i], vi = d.vel[i];
        const dvec4 c1 = d.c1[i], c2 = d.c2[i], c3 = d.c3[i];
        const double f = P.dim / P.pndSmallZero;
        forMask(d, i, d.maskS[i], [&](int j, size_t) {
            dvec4 pj = d.pos[j], vj = d.vel[j];
            PairG q = pairOf(pj, pi);
            double vx = vj.x - vi.x, vy = vj.y - vi.y, vz = vj.z - vi.z;
            double wS = wfun(sqrt(q.d2), P.reS, P.weightType);
            if (!P.gradientCorrection) {
                if (ni > P.epsilonZero) div += f * (d.pndi[j] / ni) * (vx * q.v0 + vy * q.v1 + vz * q.v2) * wS / q.d2;
            } else {
                double a0 = q.v0 * c1.x + q.v1 * c1.y + q.v2 * c1.z;
                double a1 = q.v0 * c2.x + q.v1 * c2.y + q.v2 * c2.z;
                double a2 = q.v0 * c3.x + q.v1 * c3.y + q.v2 * c3.z;
                div += f * (vx * a0 + vy * a1 + vz * a2) * wS / q.d2;
            }
        });
    }
    d.velDiv[i] = div;
}
// calcWallSlipVelDivergence / calcWallNoSlipVelDivergence, src/MpsPressure.cpp:560-790
// (rigid mesh: wall velocity 0): mirror velocity R v_i (slip) or -v_i (no-slip), the no-slip
// pair vectors reflected by R, over the near-wall fluid with n_i > eps.
__global__ void __launch_bounds__(BLK) k_wall_vel_div(Dev d) {
    int i = nearIndex(d);
    if (i < 0) return;
    const MpsParams& P = d.P;
    const double ni = d.pndi[i];
    if (!(ni > P.epsilonZero)) return;
    const bool noslip = P.slipCondition == 0;
    const dvec4 pi = d.pos[i], mi = d.mirror[i], vi = d.vel[i];
    ReflG r = makeRefl(pi, mi, P.epsilonZero, false);
    double vm[3];
    if (noslip) { vm[0] = -vi.x; vm[1] = -vi.y; vm[2] = -vi.z; }
    else {
        vm[0] = r.R[0] * vi.x + r.R[1] * vi.y + r.R[2] * vi.z;
        vm[1] = r.R[3] * vi.x + r.R[4] * vi.y + r.R[5] * vi.z;
        vm[2] = r.R[6] * vi.x + r.R[7] * vi.y + r.R[8] * vi.z;
    }
    const double f = P.dim / P.pndSmallZero;
    double div = 0.0;
    auto term = [&](double vx, double vy, double vz, double m0, double m1, double m2, double dm2, double pj) {
        double wS = wfun(sqrt(dm2), P.reS, P.weightType);
        if (noslip) {
            vx = -vx; vy = -vy; vz = -vz;
            double a0 = r.R[0] * m0 + r.R[1] * m1 + r.R[2] * m2;
            double a1 = r.R[3] * m0 + r.R[4] * m1 + r.R[5] * m2;
            double a2 = r.R[6] * m0 + r.R[7] * m1 + r.R[8] * m2;
            m0 = a0; m1 = a1; m2 = a2;
        }
        div += f * (pj / ni) * (vx * m0 + vy * m1 + vz * m2) * wS / dm2;
    };
    forNbrs(d, i, [&](int j) {
        dvec4 pj = d.pos[j];
        PairG q = pairOf(pj, pi);
        if (q.d2 < P.reS2) {
            PairM m = pairMirror(pj, mi);
            if (m.dm2 < P.reS2 && q.d2 < m.dm2) {
                dvec4 vj = d.vel[j];
                term(vj.x - vm[0], vj.y - vm[1], vj.z - vm[2], m.m0, m.m1, m.m2, m.dm2, d.pndi[j]);
            }
        }
    });
    PairM s = pairMirror(pi, mi);
    if (s.dm2 < P.reS2) term(vi.x - vm[0], vi.y - vm[1], vi.z - vm[2], s.m0, s.m1, s.m2, s.dm2, ni);
    d.velDiv[i] += div;
}
void launchVelDivergence(const Dev& d, cudaStream_t s) {
    k_vel_div<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    if (d.P.wallType == 1) k_wall_vel_div<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ correction matrix
// MpsVectorMatrix::correctionMatrix + inverseMatrix (identity when det <= eps or numNeigh < 4),
// src/MpsVectorMatrix.cpp:20-166, from the sums of w / r^2 r r^T over the reS entries.
struct Moments {
    double xx = 0, xy = 0, xz = 0, yy = 0, yz = 0, zz = 0;
    __device__ __forceinline__ void add(double v0, double v1, double v2, double wd) {
        const double t0 = wd * v0, t1 = wd * v1, t2 = wd * v2;
        xx += t0 * v0; xy += t0 * v1; xz += t0 * v2;
        yy += t1 * v1; yz += t1 * v2; zz += t2 * v2;
    }
    template <int L>
    __device__ __forceinline__ void sum() {
        xx = laneSum<L>(xx); xy = laneSum<L>(xy); xz = laneSum<L>(xz);
        yy = laneSum<L>(yy); yz = laneSum<L>(yz); zz = laneSum<L>(zz);
    }
    __device__ __forceinline__ void store(const Dev& d, int i, int numNeigh, dvec4* c1, dvec4* c2, dvec4* c3) const {
        const MpsParams& P = d.P;
        const double c = -P.coeffPressGrad;
        double m[6] = {xx * c, xy * c, xz * c, yy * c, yz * c, zz * c};
        invertSym3(m, (int)P.dim, P.epsilonZero);
        if (numNeigh < 4) {
            m[0] = m[3] = m[5] = 1.0;
            m[1] = m[2] = m[4] = 0.0;
        }
        c1[i] = make_dvec4(m[0], m[1], m[2], 0.0);
        c2[i] = make_dvec4(m[1], m[3], m[4], 0.0);
        c3[i] = make_dvec4(m[2], m[4], m[5], 0.0);
    }
};
template <int L>
__global__ void __launch_bounds__(BLK) k_corr_matrix(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const dvec4 pi = d.pos[i];
    Moments M;
    forMaskLane<L>(d, i, d.maskS[i], l, [&](int j, size_t e, int) {
        const dvec4 pj = d.pos[j];
        M.add(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z, d.cwd[e]);
    });
    M.sum<L>();
    if (l == 0) M.store(d, i, d.numNeigh[i], d.c1, d.c2, d.c3);
}
void launchCorrectionMatrix(const Dev& d, cudaStream_t s) {
#define LAUNCH(L) k_corr_matrix<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// ------------------------------------------------------------------ PND / NPCD
// MpsPndNeigh::calcPndnNeighNPCD, src/MpsPndNeigh.cpp:199-331 (init == 0), and
// setInitialPndNumberOfNeighNPCD, src/MpsPndNeigh.cpp:21-101 (init == 1).
// CORR: the correction matrix's moment sums over the reS entries in the same pass (it shares
// the entries, their gathers and their pair vectors), into the staging arrays that the
// correction-matrix operator publishes.  FP64-pipe bound: 864k particles 951 us (463 for the
// PND sums and 1,003 for the matrix when each had its own pass).
// bc: the boundary condition follows from these sums alone and is written too (the step's next
// operator).
template <int INIT, bool CORR, int L>
__global__ void __launch_bounds__(BLK) k_pnd_npcd(Dev d, bool bc) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i];
    double ni = 0.0, nx = 0.0, ny = 0.0, nz = 0.0;
    Moments M;
    const Mask mL = d.maskL[i], mS = d.maskS[i];
    forMaskLane<L>(d, i, CORR ? mS : (mL & mS), l, [&](int j, size_t e, int k) {
        const dvec4 pj = d.pos[j];
        const double v0 = pj.x - pi.x, v1 = pj.y - pi.y, v2 = pj.z - pi.z;
        if (!CORR || maskHas(mL, k)) {
            const double wS = d.cw[e];
            ni += wS;
            nx += v0 * wS; ny += v1 * wS; nz += v2 * wS;
        }
        if (CORR) M.add(v0, v1, v2, d.cwd[e]);
    });
    ni = laneSum<L>(ni); nx = laneSum<L>(nx); ny = laneSum<L>(ny); nz = laneSum<L>(nz);
    if (CORR) M.sum<L>();
    if (l != 0) return;
    int nn = (INIT ? 0 : d.nNeighWall[i]) + maskCount(mL);
    dvec4 np = INIT ? make_dvec4(0, 0, 0, 0) : d.npcd[i];
    np.x += nx; np.y += ny; np.z += nz;
    double pndSmall;
    if (INIT) {
        double pn = d.pndi[i] + ni;     // pndi accumulates onto its initial value
        pn += d.pndWall[i];
        if (d.type[i] == P.wall) pn = P.pndSmallZero;
        d.pndi[i] = pn;
        d.pndki[i] = pn;
        pndSmall = pn;
        nn += d.nNeighWall[i];
    } else {
        if (P.pndType == 0 || P.pndType == 1) {
            d.pndki[i] = d.pndi[i];
            d.pndi[i] = ni + d.pndWall[i];
        }
        pndSmall = ni + d.pndWall[i];
    }
    d.pndSmall[i] = pndSmall;
    d.numNeigh[i] = nn;
    if (ni > P.epsilonZero) { np.x /= pndSmall; np.y /= pndSmall; np.z /= pndSmall; }
    d.npcd[i] = np;
    d.npcd2[i] = np.x * np.x + np.y * np.y + np.z * np.z;
    dvec4 nw = d.polyNormal[i];
    d.devDot[i] = (np.x * nw.x + np.y * nw.y + np.z * nw.z < 0.0) ? 1.0 : -1.0;
    if (bc) d.bc[i] = boundaryCondition(d, i, pndSmall, nn, np.x * np.x + np.y * np.y + np.z * np.z);
    if (CORR) M.store(d, i, nn, d.c1n, d.c2n, d.c3n);
}
template <int INIT, bool CORR>
static void launchPndNpcd(const Dev& d, bool bc, cudaStream_t s) {
#define LAUNCH(L) k_pnd_npcd<INIT, CORR, L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d, bc)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}
void launchPndNeighNpcd(const Dev& d, cudaStream_t s, bool withCorrection, bool withBC) {
    if (withCorrection) launchPndNpcd<0, true>(d, withBC, s);
    else launchPndNpcd<0, false>(d, withBC, s);
}

// ------------------------------------------------------------------ diffusive PND (pnd type 2)
// MpsPndNeigh::calcPndDiffusiveTerm, src/MpsPndNeigh.cpp:334-489.  What is constant per
// particle (the time step and density factors, n0 and n_i) multiplies the sums once (108k
// particles: 161 -> 136 us).
template <int L>
__global__ void __launch_bounds__(BLK) k_pnd_diffusive(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const double ni = d.pndi[i];
    if (ni < P.epsilonZero) return;
    const dvec4 pi = d.pos[i], vi = d.vel[i];
    const dvec4 C1 = d.c1[i], C2 = d.c2[i], C3 = d.c3[i];
    const double Pi = d.press[i], rho = P.DNS_FL1;
    const bool fi = d.type[i] == P.fluid;
    // hydrostatic part: -2 rho rho / (rho + rho) g . r
    const double kg = -2.0 * (rho * rho / (rho + rho));
    const double gx = kg * P.gravity[0], gy = kg * P.gravity[1], gz = kg * P.gravity[2];
    double Di = 0.0, DivV = 0.0;
    const Mask mL = d.maskL[i], mS = d.maskS[i] & mL;
    const double* wLc = d.cwL ? d.cwL : d.cw;
    forMaskLane<L>(d, i, mL, l, [&](int j, size_t e, int k) {
        const dvec4 pj = d.pos[j];
        const double v0 = pj.x - pi.x, v1 = pj.y - pi.y, v2 = pj.z - pi.z;
        if (fi && d.type[j] == P.fluid) Di += (d.press[j] - Pi - (gx * v0 + gy * v1 + gz * v2)) * wLc[e];
        if (maskHas(mS, k)) {
            const dvec4 vj = d.vel[j];
            const double vx = vj.x - vi.x, vy = vj.y - vi.y, vz = vj.z - vi.z;
            const double wd = d.cwd[e];   // wS / r^2
            if (!P.gradientCorrection) {
                DivV += d.pndi[j] * (vx * v0 + vy * v1 + vz * v2) * wd;
            } else {
                const double a0 = v0 * C1.x + v1 * C1.y + v2 * C1.z;
                const double a1 = v0 * C2.x + v1 * C2.y + v2 * C2.z;
                const double a2 = v0 * C3.x + v1 * C3.y + v2 * C3.z;
                DivV += (vx * a0 + vy * a1 + vz * a2) * wd;
            }
        }
    });
    Di = laneSum<L>(Di); DivV = laneSum<L>(DivV);
    if (l != 0) return;
    Di *= P.timeStep / rho * P.coeffViscMultiphase;
    DivV *= P.dim / P.pndSmallZero;
    if (!P.gradientCorrection) DivV /= ni;
    d.aux1[i] = ni * (1.0 + P.timeStep * (-DivV + Di * 1.0));
    d.velDiv[i] = DivV;
    d.diffTerm[i] = Di;
}

// MpsPndNeigh::calcWallSlipPndDiffusiveTerm / calcWallNoSlipPndDiffusiveTerm,
// src/MpsPndNeigh.cpp:492-744 (fixed wall: wall velocity zero)
__global__ void __launch_bounds__(WALL_BLK) k_wall_pnd_diffusive(Dev d) {
    __shared__ double sm[32], R[9][32], vm[3][32];
    const MpsParams& P = d.P;
    const bool noslip = P.slipCondition == 0;
    const double cdiv = P.dim / P.pndSmallZero;
    // cdiv (n_j / n_i) (v . m) w / |m|^2, the no-slip pair vectors reflected by R
    auto term = [&](int g, double ni, double vx, double vy, double vz, const PairG& m, double wd, double nj) {
        if (!noslip) return cdiv * (nj / ni) * (vx * m.v0 + vy * m.v1 + vz * m.v2) * wd;
        const double a0 = R[0][g] * m.v0 + R[1][g] * m.v1 + R[2][g] * m.v2;
        const double a1 = R[3][g] * m.v0 + R[4][g] * m.v1 + R[5][g] * m.v2;
        const double a2 = R[6][g] * m.v0 + R[7][g] * m.v1 + R[8][g] * m.v2;
        return -(cdiv * (nj / ni) * (vx * a0 + vy * a1 + vz * a2) * wd);
    };
    forNearWall(d, [&](int i, int g) {
        const dvec4 vi = d.vel[i];
        const ReflG r = makeRefl(d.pos[i], d.mirror[i], P.epsilonZero, false);
#pragma unroll
        for (int k = 0; k < 9; k++) R[k][g] = r.R[k];
#pragma unroll
        for (int a = 0; a < 3; a++)
            vm[a][g] = noslip ? -(a == 0 ? vi.x : a == 1 ? vi.y : vi.z)
                              : r.R[3 * a] * vi.x + r.R[3 * a + 1] * vi.y + r.R[3 * a + 2] * vi.z;
    }, [&](int i, int g, int l) {
        const double ni = d.pndi[i];
        const dvec4 mi = d.mirror[i];
        double div = 0.0;
        if (ni > P.epsilonZero)
            forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorS[i], l, [&](int j, int) {
                const PairG m = pairSum(d.pos[j], mi);
                double wS, wd;
                weightR(m.d2, P.reS, P.weightType, wS, wd);
                const dvec4 vj = d.vel[j];
                div += term(g, ni, vj.x - vm[0][g], vj.y - vm[1][g], vj.z - vm[2][g], m, wd, d.pndi[j]);
            });
        div = laneSum<WALL_L>(div);
        if (l == 0) sm[g] = div;
    }, [&](int i, int g) {
        const double ni = d.pndi[i];
        if (!(ni > P.epsilonZero)) return;
        const dvec4 pi = d.pos[i], vi = d.vel[i], mi = d.mirror[i];
        double div = sm[g];
        if (pairMirror(pi, mi).dm2 < P.reS2) {
            const PairG m = pairSum(pi, mi);
            double wS, wd;
            weightR(m.d2, P.reS, P.weightType, wS, wd);
            div += term(g, ni, vi.x - vm[0][g], vi.y - vm[1][g], vi.z - vm[2][g], m, wd, ni);
        }
        d.aux1[i] += -ni * P.timeStep * div;
    });
}

// MpsPndNeigh::updatePnd, src/MpsPndNeigh.cpp:747-774
__global__ void k_update_pnd(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    d.pndi[i] = d.aux1[i];
    d.aux1[i] = 0.0;
}

// MpsPndNeigh::meanPndParticlesWallDummySurface, src/MpsPndNeigh.cpp:777-852
__global__ void __launch_bounds__(BLK) k_mean_pnd_wds(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    double up = 0.0, dn = 0.0;
    if (d.type[i] == P.wall || d.bc[i] == P.surface) {
        forMask(d, i, d.maskS[i], [&](int j, size_t e) {
            double wS = d.cw[e];
            up += d.pndi[j] * wS; dn += wS;
        });
    }
    d.aux1[i] = up; d.aux2[i] = dn;
}
__global__ void k_mean_pnd_wds_apply(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (d.type[i] == P.wall || d.bc[i] == P.surface) {
        double a1 = d.aux1[i], a2 = d.aux2[i];
        d.pndi[i] = (a2 < P.epsilonZero) ? a1 : a1 / a2;
    }
    d.aux1[i] = 0.0; d.aux2[i] = 0.0;
}

void launchPndDiffusive(const Dev& d, cudaStream_t s) {
#define LAUNCH(L) k_pnd_diffusive<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
    if (d.P.wallType == 1) k_wall_pnd_diffusive<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d);
    k_update_pnd<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    k_mean_pnd_wds<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    k_mean_pnd_wds_apply<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
}

// ------------------------------------------------------------------ mean PND (pnd type 1 and init)
// MpsPndNeigh::meanWallPnd, src/MpsPndNeigh.cpp:923-994 (sets aux1/aux2)
__global__ void __launch_bounds__(BLK) k_mean_wall_pnd(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    double up = 0.0, dn = 0.0;
    if (d.nearWall[i]) {
        dvec4 pi = d.pos[i], mi = d.mirror[i];
        forNbrs(d, i, [&](int j) {
            dvec4 pj = d.pos[j];
            PairG q = pairOf(pj, pi);
            if (q.d2 < P.reS2) {
                PairM m = pairMirror(pj, mi);
                if (m.dm2 < P.reS2 && q.d2 < m.dm2) {
                    double wS = wfun(sqrt(m.dm2), P.reS, P.weightType);
                    up += d.pndi[j] * wS; dn += wS;
                }
            }
        });
        PairM s = pairMirror(pi, mi);
        if (s.dm2 < P.reS2) {
            double wS = wfun(sqrt(s.dm2), P.reS, P.weightType);
            up += d.pndi[i] * wS; dn += wS;
        }
    }
    d.aux1[i] = up; d.aux2[i] = dn;
}
// MpsPndNeigh::meanPnd, src/MpsPndNeigh.cpp:855-920 (adds onto aux1/aux2, then divides)
__global__ void __launch_bounds__(BLK) k_mean_pnd(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    double up = 0.0, dn = 0.0;
    forMask(d, i, d.maskS[i], [&](int j, size_t e) {
        double wS = d.cw[e];
        up += d.pndi[j] * wS; dn += wS;
    });
    d.aux1[i] += up; d.aux2[i] += dn;
}
__global__ void k_mean_pnd_apply(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    double a1 = d.aux1[i], a2 = d.aux2[i];
    d.pndi[i] = (d.numNeigh[i] < 1) ? a1 : a1 / a2;
    d.aux1[i] = 0.0; d.aux2[i] = 0.0;
}
// MpsPndNeigh::meanNeighFluidPnd, src/MpsPndNeigh.cpp:997-1050
__global__ void __launch_bounds__(BLK) k_mean_neigh_fluid_pnd(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    double up = 0.0, dn = 0.0;
    forMask(d, i, d.maskS[i], [&](int j, size_t e) {
        if (d.type[j] != P.fluid) return;
        double wS = d.cw[e];
        up += d.pndki[j] * wS; dn += wS;
    });
    d.pndski[i] = (dn > P.epsilonZero) ? up / dn : up;
}
void launchPndMean(const Dev& d, cudaStream_t s) {
    if (d.P.wallType == 1) k_mean_wall_pnd<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    k_mean_pnd<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    k_mean_pnd_apply<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
}
// step-0 sequence, src/main.cpp:158-166
void launchInitPnd(const Dev& d, cudaStream_t s) {
    launchPndNpcd<1, false>(d, false, s);
    launchPndMean(d, s);
    k_mean_neigh_fluid_pnd<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ boundary condition
// MpsBoundaryCondition::updateParticleBC, types 0 and 1, src/MpsBoundaryCondition.cpp:173-204
__global__ void k_update_bc(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    d.bc[i] = boundaryCondition(d, i, d.pndSmall[i], d.numNeigh[i], d.npcd2[i]);
}
void launchUpdateBC(const Dev& d, cudaStream_t s) { k_update_bc<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }

// ------------------------------------------------------------------ ARC free surface
// MpsShifting::calcNormalParticles, src/MpsShifting.cpp:106-166: n_i = -sum r_ij w / |r_ij| / n0
// over the reS entries off the mirror side
__global__ void __launch_bounds__(BLK) k_normal(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i];
    double nx = 0, ny = 0, nz = 0;
    forMask(d, i, d.maskS[i], [&](int j, size_t) {
        PairG q = pairOf(d.pos[j], pi);
        double dst = sqrt(q.d2);
        double wS = wfun(dst, P.reS, P.weightType);
        nx += q.v0 * wS / dst; ny += q.v1 * wS / dst; nz += q.v2 * wS / dst;
    });
    d.normal[i] = make_dvec4(-nx / P.pndSmallZero, -ny / P.pndSmallZero, -nz / P.pndSmallZero, 0.0);
}
// calcWallNormalParticles, src/MpsShifting.cpp:319-420: mirror entries of the near-wall fluid
// and i as a neighbour of its mirror, reflected by R
__global__ void __launch_bounds__(BLK) k_wall_normal(Dev d) {
    int i = nearIndex(d);
    if (i < 0) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i], mi = d.mirror[i];
    ReflG r = makeRefl(pi, mi, P.epsilonZero, true);
    double dx = 0, dy = 0, dz = 0;
    forNbrs(d, i, [&](int j) {
        dvec4 pj = d.pos[j];
        PairG q = pairOf(pj, pi);
        if (q.d2 < P.reS2) {
            PairM m = pairMirror(pj, mi);
            if (m.dm2 < P.reS2 && q.d2 < m.dm2) {
                double dst = sqrt(m.dm2);
                double wS = wfun(dst, P.reS, P.weightType);
                dx += m.m0 * wS / dst; dy += m.m1 * wS / dst; dz += m.m2 * wS / dst;
            }
        }
    });
    PairM s = pairMirror(pi, mi);
    if (s.dm2 < P.reS2) {
        double dst = sqrt(s.dm2);
        double wS = wfun(dst, P.reS, P.weightType);
        dx += s.m0 * wS / dst; dy += s.m1 * wS / dst; dz += s.m2 * wS / dst;
    }
    dvec4 n = d.normal[i];
    n.x += -(r.R[0] * dx + r.R[1] * dy + r.R[2] * dz) / P.pndSmallZero;
    n.y += -(r.R[3] * dx + r.R[4] * dy + r.R[5] * dz) / P.pndSmallZero;
    n.z += -(r.R[6] * dx + r.R[7] * dy + r.R[8] * dz) / P.pndSmallZero;
    d.normal[i] = n;
}
// MpsBoundaryCondition::updateParticleBC type 2 (ARC), src/MpsBoundaryCondition.cpp:205-395:
// inner when PND, neighbour count and normal allow it; otherwise the list entries in scan
// order (the reference's bucket scan order) decide: the first real or (polygon) mirrored
// neighbour that passes the distance / angle test makes the particle inner, a tested one
// that fails makes it surface (until a later one passes); untested: the PND flag stays.
__global__ void __launch_bounds__(BLK) k_update_bc_arc(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (d.type[i] == P.dummyWall) { d.bc[i] = P.other; return; }
    int bc = (d.pndSmall[i] < P.betaPnd) ? P.surface : P.inner;
    dvec4 nv = d.normal[i];
    double n[3] = {nv.x, nv.y, nv.z};
    double norm2 = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
    if (d.pndi[i] >= P.betaPnd && d.numNeigh[i] >= P.betaNeigh && norm2 <= P.normThreshold2) {
        d.bc[i] = P.inner;
        return;
    }
    const dvec4 pi = d.pos[i], mi = d.mirror[i];
    if (norm2 > P.epsilonZero) { double q = sqrt(norm2); n[0] /= q; n[1] /= q; n[2] /= q; }
    else n[0] = n[1] = n[2] = 0.0;
    ReflG r = makeRefl(pi, mi, P.epsilonZero, false);
    double nm[3];
    for (int a = 0; a < 3; a++) nm[a] = r.R[a * 3] * n[0] + r.R[a * 3 + 1] * n[1] + r.R[a * 3 + 2] * n[2];
    double nm2 = nm[0] * nm[0] + nm[1] * nm[1] + nm[2] * nm[2];
    if (nm2 > P.epsilonZero) { double q = sqrt(nm2); nm[0] /= q; nm[1] /= q; nm[2] /= q; }
    else nm[0] = nm[1] = nm[2] = 0.0;
    const double ax = pi.x + P.partDist * n[0], ay = pi.y + P.partDist * n[1], az = pi.z + P.partDist * n[2];
    const double bx = mi.x + P.partDist * nm[0], by = mi.y + P.partDist * nm[1], bz = mi.z + P.partDist * nm[2];
    SideCtx sc = sideCtx(d, i, pi);
    const int c = d.nbrCount[i];
    const int* row = d.nbr + i;
    for (int k = 0; k < c; k++) {
        const int j = ldStream(row + (size_t)k * d.N0);
        const dvec4 pj = d.pos[j];
        PairG q = pairOf(pj, pi);
        if (!(q.d2 < P.reS2)) continue;
        if (sideOK(sc, pj, q.d2)) {
            double c0 = pj.x - ax, c1 = pj.y - ay, c2 = pj.z - az;
            double dinj2 = c0 * c0 + c1 * c1 + c2 * c2;
            double ang = acos((q.v0 * n[0] + q.v1 * n[1] + q.v2 * n[2]) / sqrt(q.d2));
            if ((q.d2 >= P.dstThreshold2 && dinj2 < P.hThreshold2) || (q.d2 < P.dstThreshold2 && ang < P.thetaArc)) {
                bc = P.inner;
                break;
            }
            bc = P.surface;
        }
        if (P.wallType == 1) {
            PairM m = pairMirror(pj, mi);
            if (m.dm2 < P.reS2 && q.d2 < m.dm2) {
                double c0 = pj.x - bx, c1 = pj.y - by, c2 = pj.z - bz;
                double dimnj2 = c0 * c0 + c1 * c1 + c2 * c2;
                double angm = acos((m.m0 * nm[0] + m.m1 * nm[1] + m.m2 * nm[2]) / sqrt(m.dm2));
                if ((m.dm2 >= P.dstThreshold2 && dimnj2 < P.hThreshold2) || (m.dm2 < P.dstThreshold2 && angm < P.thetaArc)) {
                    bc = P.inner;
                    break;
                }
                bc = P.surface;
            }
        }
    }
    d.bc[i] = bc;
}
void launchUpdateBCArc(const Dev& d, cudaStream_t s) {
    k_normal<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    if (d.P.wallType == 1) k_wall_normal<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    k_update_bc_arc<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ EOS
// MpsPressure::calcPressEMPS / calcPressWCMPS, src/MpsPressure.cpp:62-163
__global__ void k_eos(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    double mi = P.DNS_FL1;
    double p = 0.0;
    if (d.bc[i] == P.inner) {
        if (P.mpsType == 0) p = (d.pndi[i] - P.pndSmallZero) * P.coeffPressEMPS * mi;
        else p = (mi * P.coeffPressWCMPS / P.gamma) * (pow(d.pndi[i] / P.pndSmallZero, P.gamma) - 1);
    }
    if (p < 0.0) p = 0.0;
    d.press[i] = p;
}
void launchEOS(const Dev& d, cudaStream_t s) { k_eos<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }

// MpsPressure::extrapolatePressParticlesWallDummy, src/MpsPressure.cpp:792-846
template <int L>
__global__ void __launch_bounds__(BLK) k_extrapolate(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (!(d.type[i] == P.dummyWall || (P.mpsType == 1 && d.type[i] == P.wall))) return;
    const dvec4 pi = d.pos[i];
    double ni = 0.0, pr = 0.0;
    // particle walls: maskS is exactly dst^2 < reS^2 (no mirror side test)
    forMaskLane<L>(d, i, d.maskS[i], l, [&](int j, size_t e, int) {
        if (d.type[j] != P.fluid) return;
        dvec4 pj = d.pos[j];
        double v0 = pj.x - pi.x, v1 = pj.y - pi.y, v2 = pj.z - pi.z;
        double wS = d.cw[e];
        ni += wS;
        pr += (d.press[j] - P.DNS_FL1 * (P.gravity[0] * v0 + P.gravity[1] * v1 + P.gravity[2] * v2)) * wS;
    });
    ni = laneSum<L>(ni); pr = laneSum<L>(pr);
    if (pr < 0.0 || l != 0) return;
    d.press[i] = (ni > 0) ? pr / ni : pr;
}
void launchExtrapolatePress(const Dev& d, cudaStream_t s) {
#define LAUNCH(L) k_extrapolate<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// ------------------------------------------------------------------ pressure gradient
__host__ __device__ __forceinline__ bool ratioGradient(int gt) { return gt != 0 && gt != 1 && gt != 2; }
// p / n of every particle for gradient type 3 (a division per particle instead of one per pair)
__global__ void k_press_ratio(Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N0) return;
    const double n = d.pndi[i];
    d.pAux[i] = n > d.P.epsilonZero ? d.press[i] / n : 0.0;
}
// MpsPressure::calcPressGradient, src/MpsPressure.cpp:1217-1338 (p_min sweep, then sum).  The
// correction matrix, constant per particle, multiplies the sum once: sum (C r) f = C (sum r f)
// leaves 8 FP64 operations an entry for 17 (864k particles: 952 -> 450 us, type 3 at 108k:
// 386 -> 90 us).
template <int L>
__global__ void __launch_bounds__(BLK) k_press_grad(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i];
    const double Pi = d.press[i], ni = d.pndi[i];
    const int gt = P.gradientType;
    const Mask mS = d.maskS[i];
    double base = Pi;
    if (gt == 0 || gt == 2) {
        double pmin = Pi;
        forMaskLane<L>(d, i, mS, l, [&](int j, size_t, int) { minBits(pmin, d.press[j]); });
#pragma unroll
        for (int o = 1; o < L; o <<= 1) minBits(pmin, __shfl_xor_sync(laneGroup<L>(), pmin, o));
        if (l == 0) d.pAux[i] = pmin;
        base = gt == 0 ? -pmin : Pi - 2.0 * pmin;
    }
    const bool ratio = ratioGradient(gt);
    const double qi = ratio ? d.pAux[i] : 0.0;
    double ax = 0, ay = 0, az = 0;
    forMaskLane<L>(d, i, mS, l, [&](int j, size_t e, int) {
        const dvec4 pj = d.pos[j];
        double f;
        if (!ratio) f = (d.press[j] + base) * d.cwd[e];   // cwd: wS / r^2
        else {
            const double nj = d.pndi[j];
            f = (ni > P.epsilonZero && nj > P.epsilonZero) ? (ni * d.pAux[j] + nj * qi) * d.cwd[e] : d.cw[e];
        }
        ax += (pj.x - pi.x) * f; ay += (pj.y - pi.y) * f; az += (pj.z - pi.z) * f;
    });
    ax = laneSum<L>(ax); ay = laneSum<L>(ay); az = laneSum<L>(az);
    if (l != 0) return;
    if (P.gradientCorrection) {
        const dvec4 C1 = d.c1[i], C2 = d.c2[i], C3 = d.c3[i];
        const double bx = C1.x * ax + C1.y * ay + C1.z * az, by = C2.x * ax + C2.y * ay + C2.z * az,
                     bz = C3.x * ax + C3.y * ay + C3.z * az;
        ax = bx; ay = by; az = bz;
    }
    d.acc[i] = make_dvec4(d.cPG * ax, d.cPG * ay, d.cPG * az, 0.0);
}
void launchPressGradient(const Dev& d, cudaStream_t s) {
    if (ratioGradient(d.P.gradientType)) k_press_ratio<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
#define LAUNCH(L) k_press_grad<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// Wall term of the prediction's pressure gradient at a fluid particle near the polygon wall
// (Mitsume's mirror model and the repulsive force), src/MpsPressure.cpp:1031-1214: the sums
// over the candidates that forCand passes as f(j, pj, q), j != i, returned as
// fac * R a * coeffPressGrad - f_rep (fac = 1 - relax_fact).
template <class C>
__device__ __forceinline__ void wallGradTerm(const Dev& d, int i, dvec4 pi, double fac, C&& forCand, double g[3]) {
    const MpsParams& P = d.P;
    // min(velMax of the last corrector, expected maximum velocity)^2 (src/MpsPressure.cpp:1342-1344)
    double vm = fmin(*d.velMax, P.expectMaxVelocity);
    double vMax2 = vm * vm;
    dvec4 mi = d.mirror[i];
    double Pi = d.press[i], pmin = Pi, ni = d.pndi[i];
    int gt = P.gradientType;
    ReflG r = makeRefl(pi, mi, P.epsilonZero, true);
    if (gt == 0 || gt == 2) {
        forCand([&](int j, dvec4 pj, PairG q) {
            if (q.d2 < P.reS2) {
                PairM m = pairMirror(pj, mi);
                if (q.d2 < m.dm2) { double pj_ = d.press[j]; if (pmin > pj_) pmin = pj_; }
            }
        });
    }
    auto phi = [&](double Pj, double nj, double dm2, double wS) {
        if (gt == 0) return wS * ((Pj - pmin) / dm2);
        if (gt == 1) return wS * ((Pj + Pi) / dm2);
        if (gt == 2) return wS * ((Pj + Pi - 2.0 * pmin) / dm2);
        if (gt == 3 && ni > P.epsilonZero && nj > P.epsilonZero) return wS * ((ni * Pj / nj + nj * Pi / ni) / dm2);
        return wS;
    };
    double ax = 0, ay = 0, az = 0;
    forCand([&](int j, dvec4 pj, PairG q) {
        if (q.d2 < P.reS2) {
            PairM m = pairMirror(pj, mi);
            if (m.dm2 < P.reS2 && q.d2 < m.dm2) {
                double wS = wfun(sqrt(m.dm2), P.reS, P.weightType);
                wS = phi(d.press[j], d.pndi[j], m.dm2, wS);
                ax += m.m0 * wS; ay += m.m1 * wS; az += m.m2 * wS;
            }
        }
    });
    PairM s = pairMirror(pi, mi);
    if (s.dm2 < P.reS2) {
        double wS = wfun(sqrt(s.dm2), P.reS, P.weightType);
        wS = phi(Pi, ni, s.dm2, wS);
        ax += s.m0 * wS; ay += s.m1 * wS; az += s.m2 * wS;
    }
    double f[3];
    wallRepulsion(P, r, vMax2, f);
    g[0] = fac * (r.R[0] * ax + r.R[1] * ay + r.R[2] * az) * P.coeffPressGrad - f[0];
    g[1] = fac * (r.R[3] * ax + r.R[4] * ay + r.R[5] * az) * P.coeffPressGrad - f[1];
    g[2] = fac * (r.R[6] * ax + r.R[7] * ay + r.R[8] * az) * P.coeffPressGrad - f[2];
}

// MpsPressure::calcWallPressGradient + repulsive forces, src/MpsPressure.cpp:1341-1611, over
// the entry masks of the post-prediction list: p_min over the entries inside reS off the
// mirror side (maskS), the sums over the mirror entries.
// fresh: p_min of those entries is the pressure gradient's, just written (pAux); type 3 finds
// p / n there.
__global__ void __launch_bounds__(WALL_BLK) k_wall_press_grad(Dev d, bool fresh) {
    __shared__ double sm[3][32], pmn[32];
    const MpsParams& P = d.P;
    const int gt = P.gradientType;
    // min(velMax of the last corrector, expected maximum velocity)^2 (src/MpsPressure.cpp:1342-1344)
    const double vm = fmin(*d.velMax, P.expectMaxVelocity);
    // the gradient type's factor of the mirror pair, times w / |m|^2 (type 3 without PND: w)
    auto phi = [&](int i, int j, double Pi, double ni, double pmin, double wS, double wd) {
        if (gt == 0) return wd * (d.press[j] - pmin);
        if (gt == 1) return wd * (d.press[j] + Pi);
        if (gt == 2) return wd * (d.press[j] + Pi - 2.0 * pmin);
        const double nj = d.pndi[j];
        if (gt == 3 && ni > P.epsilonZero && nj > P.epsilonZero) return wd * (ni * d.pAux[j] + nj * d.pAux[i]);
        return wS;
    };
    forNearWall(d, [](int, int) {}, [&](int i, int g, int l) {
        const dvec4 mi = d.mirror[i];
        const double Pi = d.press[i], ni = d.pndi[i];
        double pmin = Pi;
        if ((gt == 0 || gt == 2) && fresh) pmin = d.pAux[i];
        else if (gt == 0 || gt == 2) {
            forMaskLane<WALL_L>(d, i, d.maskS[i], l, [&](int j, size_t, int) { minBits(pmin, d.press[j]); });
#pragma unroll
            for (int o = 1; o < WALL_L; o <<= 1) minBits(pmin, __shfl_xor_sync(laneGroup<WALL_L>(), pmin, o));
        }
        double ax = 0, ay = 0, az = 0;
        forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorS[i], l, [&](int j, int) {
            const PairG m = pairSum(d.pos[j], mi);
            double wS, wd;
            weightR(m.d2, P.reS, P.weightType, wS, wd);
            const double f = phi(i, j, Pi, ni, pmin, wS, wd);
            ax += m.v0 * f; ay += m.v1 * f; az += m.v2 * f;
        });
        ax = laneSum<WALL_L>(ax); ay = laneSum<WALL_L>(ay); az = laneSum<WALL_L>(az);
        if (l == 0) { sm[0][g] = ax; sm[1][g] = ay; sm[2][g] = az; pmn[g] = pmin; }
    }, [&](int i, int g) {
        const dvec4 pi = d.pos[i], mi = d.mirror[i];
        const double Pi = d.press[i], ni = d.pndi[i];
        const ReflG r = makeRefl(pi, mi, P.epsilonZero, true);
        double ax = sm[0][g], ay = sm[1][g], az = sm[2][g];
        if (pairMirror(pi, mi).dm2 < P.reS2) {
            const PairG m = pairSum(pi, mi);
            double wS, wd;
            weightR(m.d2, P.reS, P.weightType, wS, wd);
            if (!(m.d2 > 0.0)) wS = wfun(0.0, P.reS, P.weightType);   // on the wall: 1 / r does not give w
            const double f = phi(i, i, Pi, ni, pmn[g], wS, wd);
            ax += m.v0 * f; ay += m.v1 * f; az += m.v2 * f;
        }
        double fr[3];
        wallRepulsion(P, r, vm * vm, fr);
        double gr[3];
#pragma unroll
        for (int a = 0; a < 3; a++)
            gr[a] = P.relaxPress * (r.R[3 * a] * ax + r.R[3 * a + 1] * ay + r.R[3 * a + 2] * az) * P.coeffPressGrad - fr[a];
        dvec4 a = d.acc[i];
        a.x += gr[0] / P.DNS_FL1; a.y += gr[1] / P.DNS_FL1; a.z += gr[2] / P.DNS_FL1;
        d.acc[i] = a;
        const double vf = (P.dim == 3) ? P.partDist * P.partDist * P.partDist : P.partDist * P.partDist;
        dvec4 fw = d.forceWall[i];
        fw.x += -gr[0] * vf; fw.y += -gr[1] * vf; fw.z += -gr[2] * vf;
        d.forceWall[i] = fw;
    });
}
void launchWallPressGradient(const Dev& d, cudaStream_t s, bool fresh) {
    if (d.P.wallType != 1) return;
    if (d.P.gradientType == 3 && !fresh) k_press_ratio<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    k_wall_press_grad<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d, fresh);
}

// ------------------------------------------------------------------ prediction-step pressure gradient
// relax_fact < 1 (src/main.cpp:271-276): before the prediction, (1 - relax_fact) of the
// previous pressure's gradient at the start-of-step positions is added to the
// acceleration.  The candidates of i in scan order: the start-of-step skin list when it
// is built for these positions (its entries within the FP32 band of the ball are the
// candidates the 27-bucket scan passes to the exact FP64 test), else the scan itself.
template <class F>
__device__ __forceinline__ void forStartCandidates(const Dev& d, int i, dvec4 pi, float hi, bool skin, F&& f) {
    const float4 fi = d.posf[i];
    const int c = skin ? d.skinCnt[i] : d.K + 1;
    if (c <= d.K) {
        const int* row = d.skinNbr + i;
        for (int k = 0; k < c; k++) {
            const int j = ldStream(row + (size_t)k * d.N0);
            const float4 fj = d.posf[j];
            const float ex = fj.x - fi.x, ey = fj.y - fi.y, ez = fj.z - fi.z;
            if (ex * ex + ey * ey + ez * ez > hi) continue;
            const dvec4 pj = d.pos[j];
            f(j, pj, pairOf(pj, pi));
        }
    } else {
        forCellsNear(d, pi, fi, hi, [&](int j, dvec4 pj, PairG q) {
            if (j != i) f(j, pj, q);
        });
    }
}

// MpsPressure::predictionPressGradient, src/MpsPressure.cpp:932-1028: every particle, the
// gradient type's pair term without the correction matrix, in the reference's operation
// order (w(r) from |r|, then times (...)/r^2).
__global__ void __launch_bounds__(BLK) k_pred_press_grad(Dev d, bool skin) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i];
    const SideCtx sc = sideCtx(d, i, pi);
    const double Pi = d.press[i], ni = d.pndi[i];
    double pmin = Pi;
    const int gt = P.gradientType;
    if (gt == 0 || gt == 2) {
        forStartCandidates(d, i, pi, d.bandHiS, skin, [&](int j, dvec4 pj, PairG q) {
            if (q.d2 < P.reS2 && sideOK(sc, pj, q.d2)) { double pj_ = d.press[j]; if (pmin > pj_) pmin = pj_; }
        });
    }
    double ax = 0, ay = 0, az = 0;
    forStartCandidates(d, i, pi, d.bandHiS, skin, [&](int j, dvec4 pj, PairG q) {
        if (!(q.d2 < P.reS2) || !sideOK(sc, pj, q.d2)) return;
        double wS = wfun(sqrt(q.d2), P.reS, P.weightType);
        const double Pj = d.press[j];
        if (gt == 0) wS *= (Pj - pmin) / q.d2;
        else if (gt == 1) wS *= (Pj + Pi) / q.d2;
        else if (gt == 2) wS *= (Pj + Pi - 2.0 * pmin) / q.d2;
        else if (gt == 3) {
            const double nj = d.pndi[j];
            if (ni > P.epsilonZero && nj > P.epsilonZero) wS *= (ni * Pj / nj + nj * Pi / ni) / q.d2;
        }
        ax += q.v0 * wS; ay += q.v1 * wS; az += q.v2 * wS;
    });
    const double fac = 1.0 - P.relaxPress;
    dvec4 a = d.acc[i];
    a.x += fac * ax * P.coeffPressGrad / P.DNS_FL1;
    a.y += fac * ay * P.coeffPressGrad / P.DNS_FL1;
    a.z += fac * az * P.coeffPressGrad / P.DNS_FL1;
    d.acc[i] = a;
}

// MpsPressure::predictionWallPressGradient, src/MpsPressure.cpp:1031-1214: fluid particles
// flagged near the wall by the last wall pass (its flags and mirror positions are still
// held: the prediction resets them after this sweep), no force on the wall.
__global__ void __launch_bounds__(BLK) k_pred_wall_press_grad(Dev d, bool skin) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (d.type[i] != P.fluid || !d.nearWall[i]) return;
    const dvec4 pi = d.pos[i];
    double g[3];
    wallGradTerm(d, i, pi, 1.0 - P.relaxPress, [&](auto&& f) {
        forStartCandidates(d, i, pi, d.bandHiS, skin, f);
    }, g);
    dvec4 a = d.acc[i];
    a.x += g[0] / P.DNS_FL1; a.y += g[1] / P.DNS_FL1; a.z += g[2] / P.DNS_FL1;
    d.acc[i] = a;
}

void launchPredictPressGradient(const Dev& d, bool skin, cudaStream_t s) {
    k_pred_press_grad<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, skin);
    // the wall sweep reads the accelerations the particle sweep has completed
    if (d.P.wallType == 1) k_pred_wall_press_grad<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, skin);
}

// ------------------------------------------------------------------ wall viscosity
// MpsViscosity::calcWallNoSlipViscosity / calcWallSlipViscosity (Newtonian, fixed wall),
// src/MpsViscosity.cpp:1527-1910
__device__ __forceinline__ void wallViscMatrix(const MpsParams& P, dvec4 pi, dvec4 mi, double M[9]) {
    if (P.slipCondition == 0) {   // no-slip: -I
#pragma unroll
        for (int k = 0; k < 9; k++) M[k] = (k % 4 == 0) ? -1.0 : 0.0;
        return;
    }
    const ReflG r = makeRefl(pi, mi, P.epsilonZero, false);
#pragma unroll
    for (int k = 0; k < 9; k++) M[k] = r.R[k];
}
__global__ void __launch_bounds__(WALL_BLK) k_wall_visc(Dev d) {
    __shared__ double sm[3][32], vm[3][32];
    const MpsParams& P = d.P;
    const double mu = P.KNM_VS1 * P.DNS_FL1;
    const double neu = ((mu + mu) > P.epsilonZero ? 2.0 * mu * mu / (mu + mu) : 0.0) / P.DNS_FL1;
    forNearWall(d, [&](int i, int g) {
        const dvec4 vi = d.vel[i];
        double M[9];
        wallViscMatrix(P, d.pos[i], d.mirror[i], M);
#pragma unroll
        for (int a = 0; a < 3; a++) vm[a][g] = M[3 * a] * vi.x + M[3 * a + 1] * vi.y + M[3 * a + 2] * vi.z;
    }, [&](int i, int g, int l) {
        const dvec4 mi = d.mirror[i];
        double ax = 0, ay = 0, az = 0;
        forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorL[i], l, [&](int j, int) {
            double wL, wd;
            weightR(pairSum(d.pos[j], mi).d2, P.reL, P.weightType, wL, wd);
            const dvec4 vj = d.vel[j];
            const double f = wL * neu;
            ax += (vj.x - vm[0][g]) * f; ay += (vj.y - vm[1][g]) * f; az += (vj.z - vm[2][g]) * f;
        });
        ax = laneSum<WALL_L>(ax); ay = laneSum<WALL_L>(ay); az = laneSum<WALL_L>(az);
        if (l == 0) { sm[0][g] = ax; sm[1][g] = ay; sm[2][g] = az; }
    }, [&](int i, int g) {
        const dvec4 pi = d.pos[i], vi = d.vel[i], mi = d.mirror[i];
        double M[9];
        wallViscMatrix(P, pi, mi, M);
        double ax = sm[0][g], ay = sm[1][g], az = sm[2][g];
        PairM s = pairMirror(pi, mi);
        if (s.dm2 < P.reL2) {
            double wL = wfun(sqrt(s.dm2), P.reL, P.weightType);
            double neuS = (mu > P.epsilonZero ? 2.0 * mu * mu / (mu + mu) : 0.0) / P.DNS_FL1;
            ax += (vi.x - vm[0][g]) * wL * neuS;
            ay += (vi.y - vm[1][g]) * wL * neuS;
            az += (vi.z - vm[2][g]) * wL * neuS;
        }
        double f0 = (M[0] * ax + M[1] * ay + M[2] * az) * P.coeffViscMultiphase;
        double f1 = (M[3] * ax + M[4] * ay + M[5] * az) * P.coeffViscMultiphase;
        double f2 = (M[6] * ax + M[7] * ay + M[8] * az) * P.coeffViscMultiphase;
        dvec4 a = d.acc[i];
        a.x += f0; a.y += f1; a.z += f2;
        d.acc[i] = a;
        double vf = (P.dim == 3) ? P.partDist * P.partDist * P.partDist : P.partDist * P.partDist;
        dvec4 fw = d.forceWall[i];
        fw.x += -f0 * vf * P.DNS_FL1; fw.y += -f1 * vf * P.DNS_FL1; fw.z += -f2 * vf * P.DNS_FL1;
        d.forceWall[i] = fw;
    });
}
void launchWallViscosity(const Dev& d, cudaStream_t s) {
    if (d.P.wallType != 1) return;
    k_wall_visc<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ corrector
// MpsParticleVelPos::correctionVelocityPosition, src/MpsParticleVelPos.cpp:53-97, with the
// maximum fluid speed reduced on the device (max is order independent).  The squares are reduced,
// by their bits (a NaN is left out, as fmax leaves it), and the root is taken once per block:
// sqrt is monotone, so it is the maximum of the roots, and one per particle was most of the
// kernel's FP64 operations (864k particles, cold cache: 42.3 us, now 24.6; 6.9k: 5.9, now 4.9).
__device__ __forceinline__ unsigned long long warpMax64(unsigned long long v) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
    return ((unsigned long long)hi << 32) | lo;
}
__global__ void k_correct(Dev d, double* next) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *d.velMax = 0.0;   // the last step's value, read before; the next call's slot
    const MpsParams& P = d.P;
    unsigned long long v = 0ull;
    if (i < liveN(d) && d.type[i] == P.fluid) {
        dvec4 u = d.vel[i], a = d.acc[i], x = d.pos[i];
        double dt = P.timeStep, dt2 = P.timeStep * P.timeStep;
        u.x += a.x * dt; u.y += a.y * dt; u.z += a.z * dt;
        x.x += a.x * dt2; x.y += a.y * dt2; x.z += a.z * dt2;
        d.vel[i] = u; d.pos[i] = x;
        d.acc[i] = make_dvec4(0, 0, 0, 0);
        v = (unsigned long long)__double_as_longlong(u.x * u.x + u.y * u.y + u.z * u.z);
        if (v > 0x7ff0000000000000ull) v = 0ull;
    }
    v = warpMax64(v);
    __shared__ unsigned long long sm[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sm[w] = v;
    __syncthreads();
    if (w == 0) {
        v = warpMax64(lane < (int)(blockDim.x >> 5) ? sm[lane] : 0ull);
        if (lane == 0 && v)
            atomicMax((unsigned long long*)next,
                      (unsigned long long)__double_as_longlong(sqrt(__longlong_as_double((long long)v))));
    }
}
void launchCorrect(const Dev& d, double* next, cudaStream_t s) {
    k_correct<<<gridFor(d.N0, 256), 256, 0, s>>>(d, next);
}

// ------------------------------------------------------------------ shifting
// MpsShifting::calcShifting (type 1), src/MpsShifting.cpp:23-101: dv from the
// pre-shift velocities, then applied.
// Common head of the post-corrector scans: prefilter band of the reS ball, exact FP64
// radius and mirror-side tests; particles the sweep does not update skip the scan.
struct E2Base {
    struct Core { SideCtx sc; bool on; };
    __device__ static void start(const Dev& d, int i, Core& c, bool on) {
        c.on = on;
        if (on) c.sc = sideCtx(d, i, d.pos[i]);
    }
    __device__ static bool accept(const Dev& d, const Core& c, dvec4 pj, PairG q) {
        return q.d2 < d.P.reS2 && sideOK(c.sc, pj, q.d2);
    }
};
#define E2_COMMON \
    __device__ float hi(const Dev& d) const { return d.bandHiS; } \
    __device__ bool active(const Dev&, const State& st) const { return st.c.on; }
struct OpShiftVel {
    struct State { E2Base::Core c; dvec4 vi; double ux, uy, uz; };
    E2_COMMON
    __device__ void begin(const Dev& d, int i, State& st) const {
        E2Base::start(d, i, st.c, d.type[i] == d.P.fluid);
        st.vi = d.vel[i]; st.ux = st.uy = st.uz = 0.0;
    }
    __device__ void visit(const Dev& d, int i, State& st, int j, dvec4 pj, PairG q) const {
        if (E2Base::accept(d, st.c, pj, q)) add(d, st, j, q.d2);
    }
    __device__ __forceinline__ void add(const Dev& d, State& st, int j, double d2) const {
        double dw = dwfun(sqrt(d2), d.P.reS, d.P.weightType);
        dvec4 vj = d.vel[j];
        st.ux += dw * (vj.x - st.vi.x); st.uy += dw * (vj.y - st.vi.y); st.uz += dw * (vj.z - st.vi.z);
    }
    __device__ void end(const Dev& d, int i, State& st) const {
        bool apply = st.c.on && d.bc[i] == d.P.inner;
        d.shift[i] = apply ? make_dvec4(st.ux, st.uy, st.uz, 0.0) : make_dvec4(0, 0, 0, 0);
    }
};
__global__ void k_shift_vel_apply(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    dvec4 v = d.vel[i], du = d.shift[i];
    double c = d.P.coeffShifting1;
    v.x -= c * du.x; v.y -= c * du.y; v.z -= c * du.z;
    d.vel[i] = v;
}
// MpsShifting::calcConcAndConcGradient, src/MpsShifting.cpp:432-575: concentration, then
// gradient and position shift (each sweep reads the positions it started with).
struct OpConc {
    struct State { E2Base::Core c; double sum; };
    E2_COMMON
    __device__ void begin(const Dev& d, int i, State& st) const { E2Base::start(d, i, st.c, true); st.sum = 0.0; }
    __device__ void visit(const Dev& d, int i, State& st, int j, dvec4 pj, PairG q) const {
        if (!E2Base::accept(d, st.c, pj, q)) return;
        double w, wd;
        weightR(q.d2, d.P.reS, d.P.weightType, w, wd);
        st.sum += w;
    }
    __device__ void end(const Dev& d, int i, State& st) const {
        d.conc[i] = (st.sum + d.pndWall[i]) / d.P.pndSmallZero;
    }
};
struct OpGradConc {
    struct State { E2Base::Core c; double ci, gx, gy, gz; };
    E2_COMMON
    __device__ void begin(const Dev& d, int i, State& st) const {
        E2Base::start(d, i, st.c, d.type[i] == d.P.fluid);
        st.ci = d.conc[i]; st.gx = st.gy = st.gz = 0.0;
    }
    __device__ void visit(const Dev& d, int i, State& st, int j, dvec4 pj, PairG q) const {
        if (!E2Base::accept(d, st.c, pj, q)) return;
        double wS, wd;
        weightR(q.d2, d.P.reS, d.P.weightType, wS, wd);
        double cc = (st.ci + d.conc[j]) * wd;
        st.gx += cc * q.v0; st.gy += cc * q.v1; st.gz += cc * q.v2;
    }
    __device__ void end(const Dev& d, int i, State& st) const {
        const MpsParams& P = d.P;
        dvec4 sh = make_dvec4(0, 0, 0, 0);
        if (st.c.on) {
            double gx = st.gx * -P.coeffPressGrad, gy = st.gy * -P.coeffPressGrad, gz = st.gz * -P.coeffPressGrad;
            d.gradC[i] = make_dvec4(gx, gy, gz, 0.0);
            if (d.bc[i] == P.inner)
                sh = make_dvec4(-P.coeffShifting2 * gx, -P.coeffShifting2 * gy, -P.coeffShifting2 * gz, 0.0);
        }
        d.shift[i] = sh;
    }
};
// MpsShifting::calcWallConcAndConcGradient, src/MpsShifting.cpp:578-691, at the shifted
// positions: 40 us at 108k particles (449 as a 27-bucket FP64 scan of one thread each; float-
// float at 2.8M 427 -> 218).
__global__ void __launch_bounds__(WALL_BLK) k_wall_grad_conc(Dev d, bool skin) {
    __shared__ WallCand W;
    __shared__ double sm[3][32];
    const MpsParams& P = d.P;
    const int nn = *d.nearCount;
    const bool useSkin = skin && !*(volatile int*)d.skinFlag;
    for (int base = blockIdx.x * 32; base < nn; base += gridDim.x * 32) {
        wallCandidates(d, W, base, nn, useSkin);
        __syncthreads();
        const int g = threadIdx.x / WALL_L, l = threadIdx.x & (WALL_L - 1);
        if (base + g < nn) {
            const int i = d.nearList[base + g];
            const dvec4 mi = d.mirror[i];
            const double ci = d.conc[i];
            double dx = 0, dy = 0, dz = 0;
            forWallCand(d, W, i, g, l, [&](int j) {
                const PairG m = pairSum(d.pos[j], mi);
                double wS, wd;
                weightR(m.d2, P.reS, P.weightType, wS, wd);
                const double cc = (ci + d.conc[j]) * wd;
                dx += cc * m.v0; dy += cc * m.v1; dz += cc * m.v2;
            });
            dx = laneSum<WALL_L>(dx); dy = laneSum<WALL_L>(dy); dz = laneSum<WALL_L>(dz);
            if (l == 0) { sm[0][g] = dx; sm[1][g] = dy; sm[2][g] = dz; }
        }
        __syncthreads();
        if (threadIdx.x < 32 && base + (int)threadIdx.x < nn)
            wallGradConcEnd(d, d.nearList[base + threadIdx.x], sm[0][threadIdx.x], sm[1][threadIdx.x], sm[2][threadIdx.x]);
        __syncthreads();
    }
}
// x += shift; the FP32 copy follows the new positions (next prefiltered scan)
__device__ __forceinline__ void applyShift(const Dev& d, int i) {
    dvec4 x = d.pos[i], s = d.shift[i];
    x.x += s.x; x.y += s.y; x.z += s.z;
    d.pos[i] = x;
    float4 hi, lo;
    splitPos(x, d.P, hi, lo);
    d.posf[i] = hi;
    d.posLo[i] = lo;
}
__global__ void k_apply_shift(Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < liveN(d)) applyShift(d, i);
}
// the same for the particles near the wall
__global__ void k_apply_shift_near(Dev d) {
    const int n = *d.nearCount;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) applyShift(d, d.nearList[t]);
}
void launchShiftVelApply(const Dev& d, cudaStream_t s) { k_shift_vel_apply<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }
void launchApplyShift(const Dev& d, cudaStream_t s) { k_apply_shift<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }
void launchApplyShiftNear(const Dev& d, cudaStream_t s) {
    const int grid = gridFor(d.N0, 256) < 608 ? gridFor(d.N0, 256) : 608;
    k_apply_shift_near<<<grid, 256, 0, s>>>(d);
}
// The 27-bucket sweeps over the list of the post-corrector positions instead: its maskS
// entries (inside reS, off the mirror side) are the scan's neighbours in the scan's order.
template <int L>
__global__ void __launch_bounds__(128) k_shift_vel_list(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const OpShiftVel op;
    OpShiftVel::State st;
    const bool on = d.type[i] == d.P.fluid;
    st.c.on = on;
    st.vi = d.vel[i]; st.ux = st.uy = st.uz = 0.0;
    const dvec4 pi = d.pos[i];
    if (on) forMaskLane<L>(d, i, d.maskS[i], l, [&](int j, size_t, int) { op.add(d, st, j, pairSum(d.pos[j], pi).d2); });
    st.ux = laneSum<L>(st.ux); st.uy = laneSum<L>(st.uy); st.uz = laneSum<L>(st.uz);
    if (l == 0) op.end(d, i, st);
}
template <int L>
__global__ void __launch_bounds__(128) k_conc_list(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    double sum = 0.0;
    forMaskLane<L>(d, i, d.maskS[i], l, [&](int, size_t e, int) { sum += d.cw[e]; });
    sum = laneSum<L>(sum);
    if (l == 0) d.conc[i] = (sum + d.pndWall[i]) / d.P.pndSmallZero;
}
template <int L>
__global__ void __launch_bounds__(128) k_grad_conc_list(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    OpGradConc::State st;
    st.c.on = d.type[i] == d.P.fluid;
    st.ci = d.conc[i]; st.gx = st.gy = st.gz = 0.0;
    const dvec4 pi = d.pos[i];
    if (st.c.on)
        forMaskLane<L>(d, i, d.maskS[i], l, [&](int j, size_t e, int) {
            const dvec4 pj = d.pos[j];
            const double cc = (st.ci + d.conc[j]) * d.cwd[e];
            st.gx += cc * (pj.x - pi.x); st.gy += cc * (pj.y - pi.y); st.gz += cc * (pj.z - pi.z);
        });
    st.gx = laneSum<L>(st.gx); st.gy = laneSum<L>(st.gy); st.gz = laneSum<L>(st.gz);
    if (l == 0) OpGradConc().end(d, i, st);
}

// list: the sweeps read the list of the post-corrector positions with its weights and masks,
// filtered from the kept start-of-step skin list just before (108k particles: concentration
// and gradient 22 + 67 us beside a filter of 130, for 165 + 210 with the weights formed in
// each beside one of 24); else they scan the buckets
void launchShifting(const Dev& d, cudaStream_t s, bool list) {
    const MpsParams& P = d.P;
    if (P.shiftingType != 1 && P.shiftingType != 2) return;
    if (!list) launchPosf(d, s);   // post-corrector positions
#define LAUNCH_VEL(L) k_shift_vel_list<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d)
#define LAUNCH_CONC(L)                                          \
    k_conc_list<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d);   \
    k_grad_conc_list<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d)
    if (P.shiftingType == 1) {
        if (list) MPS_FOR_LANES(d.N0, LAUNCH_VEL);
        else launchScan(d, OpShiftVel(), s);
        k_shift_vel_apply<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    } else {
        if (list) MPS_FOR_LANES(d.N0, LAUNCH_CONC);
        else {
            launchScan(d, OpConc(), s);
            launchScan(d, OpGradConc(), s);
        }
        k_apply_shift<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
        if (P.wallType == 1) {   // the wall sweep sees the shifted positions
            if (list) launchSkinCheck(d, s, false);
            else launchNearList(d, s);
            k_wall_grad_conc<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d, list);
            launchApplyShiftNear(d, s);
        }
    }
#undef LAUNCH_VEL
#undef LAUNCH_CONC
}

// ------------------------------------------------------------------ dummy velocity
// MpsParticleVelPos::updateVelocityParticlesWallDummy, src/MpsParticleVelPos.cpp:100-158
// (dummy particles read fluid velocities only, so the update is race free in place).  L lanes per
// particle test a bucket row's candidates by their FP32 copies and sum those inside.
template <int L>
__global__ void __launch_bounds__(BLK) k_dummy_vel(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (d.type[i] != P.dummyWall) return;
    const dvec4 pi = d.pos[i];
    const float4 fi = d.posf[i];
    double ni = 0.0, ux = 0, uy = 0, uz = 0;
    int ix, iy, iz;
    bucketCoordsHi(d, pi, fi, ix, iy, iz);
    const int minZ = (iz - 1) * d.dz3, maxZ = (iz + 1) * d.dz3;
    for (int jz = minZ; jz <= maxZ; jz++)
        for (int jy = iy - 1; jy <= iy + 1; jy++) {
            const long long jb = (long long)jz * P.numBucketsXY + (long long)jy * P.numBucketsX + ix;
            const long long lo = jb - 1 > 0 ? jb - 1 : 0, hi = jb + 1 < d.nB - 1 ? jb + 1 : d.nB - 1;
            if (lo > hi) continue;
            const int s1 = d.cellStart[hi + 1];
            for (int s0 = d.cellStart[lo]; s0 < s1; s0 += 32) {
                unsigned m = 0u;
#pragma unroll 4
                for (int t = l; t < 32; t += L) {
                    if (s0 + t >= s1) break;
                    const int j = __ldg(d.cellSorted + s0 + t);
                    if (d.type[j] != P.fluid || j == i) continue;
                    if (insideF(d, dist2f(__ldg(&d.posf[j]), fi), d.bandLoL, d.bandHiL, P.reL2, i, j)) m |= 1u << t;
                }
                for (; m; m &= m - 1u) {
                    const int j = __ldg(d.cellSorted + s0 + __ffs((int)m) - 1);
                    double wL, wd;
                    weightR(pairSum(d.pos[j], pi).d2, P.reL, P.weightType, wL, wd);
                    const dvec4 vj = d.vel[j];
                    ni += wL;
                    ux += vj.x * wL; uy += vj.y * wL; uz += vj.z * wL;
                }
            }
        }
    ni = laneSum<L>(ni); ux = laneSum<L>(ux); uy = laneSum<L>(uy); uz = laneSum<L>(uz);
    if (l != 0) return;
    dvec4 v;
    if (ni > P.epsilonZero) v = make_dvec4(2.0 * 0.0 - ux / ni, 2.0 * 0.0 - uy / ni, 2.0 * 0.0 - uz / ni, 0.0);
    else v = make_dvec4(2.0 * 0.0 - ux, 2.0 * 0.0 - uy, 2.0 * 0.0 - uz, 0.0);
    d.vel[i] = v;
}
void launchDummyVelocity(const Dev& d, cudaStream_t s) {
    if (d.P.wallType != 0) return;
    launchPosfOnly(d, s);
#define LAUNCH(L) k_dummy_vel<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}
