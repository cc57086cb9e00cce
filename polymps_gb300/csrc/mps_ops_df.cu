// mps_ops_df.cu — the DF32 precision tier of the neighbour sweeps on sm_103a.
//
// Same operators, same reference order and same discrete decisions as mps_ops.cu, with
// the per-pair arithmetic in float-float (mps_df.cuh) instead of FP64: pair vectors come
// from the hi/lo position copies, weights are recomputed per entry from the float-float
// squared distance (no per-entry weight cache: FP32 work is cheaper than its HBM traffic),
// sums are float-float and each particle's result is assembled in FP64 once.  Radius and
// mirror-side decisions whose float-float value lies within the error margin fall back to
// the reference's FP64 expression, so entry sets, masks and flags equal the FP64 tier's.
#include "mps_df.cuh"
#include "mps_internal.h"
#include "mps_lanes.cuh"

#define BLK 128

// ------------------------------------------------------------------ copies
__global__ void k_df_vel(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N0) return;
    dvec4 v = d.vel[i];
    const df x = dfD(v.x), y = dfD(v.y), z = dfD(v.z);
    d.velHi[i] = make_float4(x.h, y.h, z.h, 0.f);
    d.velLo[i] = make_float4(x.l, y.l, z.l, 0.f);
}
__global__ void k_df_press(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N0) return;
    df p = dfD(d.press[i]);
    d.pressDF[i] = make_float2(p.h, p.l);
}
static void launchVelDF(const Dev& d, cudaStream_t s) { k_df_vel<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }
static void launchPressDF(const Dev& d, cudaStream_t s) { k_df_press<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }

__device__ __forceinline__ df K(float2 v) { return {v.x, v.y}; }
__device__ __forceinline__ df loadDF(const float2* p, int j) {
    float2 v = __ldg(p + j);
    return {v.x, v.y};
}

template <int L>
__device__ __forceinline__ df laneSumDF(df v) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
        const df q = {__shfl_xor_sync(laneGroup<L>(), v.h, o), __shfl_xor_sync(laneGroup<L>(), v.l, o)};
        v += q;
    }
    return v;
}
// What a pair needs of its neighbour: the position's hi and lo parts (and X, the sweep's own).
struct NbrPos {
    float4 h, l;
};
__device__ __forceinline__ NbrPos loadPos(const Dev& d, int j) { return {__ldg(&d.posf[j]), __ldg(&d.posLo[j])}; }

// ------------------------------------------------------------------ viscosity
// MpsViscosity::calcViscosity, src/MpsViscosity.cpp:20-100, at the start-of-step
// positions through the 27 buckets (Newtonian: uniform MEU and RHO).  Two phases per
// batch: the FP32 prefilter compacts the surviving slots of the thread's candidates into
// its shared-memory column (bucket order kept), then the float-float pair work runs over
// the compacted slots, so the lanes of a warp stay converged through the expensive part.
#define VCAP 48
#define VBLK 128
template <bool STRAY>
__global__ void __launch_bounds__(VBLK) k_visc_df(Dev d) {
    __shared__ int slots[VCAP * VBLK];
    const int t = threadIdx.x;
    const int i = scanParticle<STRAY>(d);
    if (i < 0) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i];
    const float4 hi = d.posf[i], li = d.posLo[i];
    const float4 vh = d.velHi[i], vl = d.velLo[i];
    const SideDF sc = sideDF(d, i, pi);
    const df R2 = K(d.k.reL2), neuW = K(d.k.neuW), neuF = K(d.k.neuF);
    const RadiusDF RL = {K(d.k.reL), K(d.k.invReL)};
    const float band = d.bandHiL;
    df ax = dfF(0.f), ay = dfF(0.f), az = dfF(0.f);
    int ix, iy, iz;
    bucketCoordsHi(d, pi, hi, ix, iy, iz);
    const int dz = (int)(P.dim - 2.0);
    const int nbk = dz ? 27 : 9;
    int bk = 0, s = 0, s1 = 0;
    bool more = true;
    while (more) {
        int n = 0;
        while (n < VCAP) {
            if (s >= s1) {
                if (bk >= nbk) { more = false; break; }
                int kz = bk / 9, ky = (bk / 3) % 3, kx = bk % 3;
                bk++;
                long long jb = (long long)((iz - 1) * dz + kz) * P.numBucketsXY +
                               (long long)(iy - 1 + ky) * P.numBucketsX + (ix - 1 + kx);
                if (jb < 0 || jb >= d.nB) continue;
                s = d.cellStart[jb];
                s1 = d.cellStart[jb + 1];
                continue;
            }
            float4 fj = __ldg(&d.posfCell[s]);
            float ex = fj.x - hi.x, ey = fj.y - hi.y, ez = fj.z - hi.z;
            if (ex * ex + ey * ey + ez * ez <= band) slots[n++ * VBLK + t] = s;
            s++;
        }
        for (int k = 0; k < n; k++) {
            const int sk = slots[k * VBLK + t];
            const int j = __ldg(d.cellSorted + sk);
            if (j == i) continue;
            const float4 hj = __ldg(&d.posfCell[sk]), lj = __ldg(&d.posLoCell[sk]);
            PairF q = pairDF(hj, lj, hi, li);
            if (!inBallDF(d, q.d2, R2, d.mgL, P.reL2, i, j)) continue;
            if (!sideOkDF(d, sc, hj, lj, q.d2, i, j)) continue;
            WeightDF w = weightDF(q.d2, RL, P.weightType);
            df c = w.w * ((d.type[j] == P.wall) ? neuW : neuF);
            float4 vhj = d.velHi[j], vlj = d.velLo[j];
            mac(ax, diffDF(vhj.x, vlj.x, vh.x, vl.x), c);
            mac(ay, diffDF(vhj.y, vlj.y, vh.y, vl.y), c);
            mac(az, diffDF(vhj.z, vlj.z, vh.z, vl.z), c);
        }
    }
    double cv = P.coeffViscMultiphase;
    d.acc[i] = make_dvec4(cv * dD(ax), cv * dD(ay), cv * dD(az), 0.0);
}
void launchViscosityDF(const Dev& d, cudaStream_t s) {
    launchVelDF(d, s);
    k_visc_df<false><<<gridFor(d.N0, VBLK), VBLK, 0, s>>>(d);
    k_visc_df<true><<<gridFor(d.N0, VBLK), VBLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ collision
// MpsParticleCollision::checkParticleCollisions, src/MpsParticleCollision.cpp:22-119.
// The sign test fDT > 0 is decided in float-float outside a margin that bounds the
// difference from the FP64 value, and in FP64 inside it.
__global__ void __launch_bounds__(BLK) k_collision_df(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    df dvx = dfF(0.f), dvy = dfF(0.f), dvz = dfF(0.f);
    bool any = false;
    if (d.type[i] == P.fluid) {
        dvec4 pi = d.pos[i];
        float4 hi = d.posf[i], li = d.posLo[i];
        float4 vh = d.velHi[i], vl = d.velLo[i];
        float vin = fabsf(vh.x) + fabsf(vh.y) + fabsf(vh.z);
        const SideDF sc = d.mirrorFar ? SideDF{} : sideDF(d, i, pi);   // {}: no side test
        const df R2 = K(d.k.coll2), cF = K(d.k.collF), cW = K(d.k.collW);
        forNbrsPosf(d, i, [&](int j, float4 hj) {
            // FP32 prefilter: most list entries lie beyond the collision distance
            const float ex = hj.x - hi.x, ey = hj.y - hi.y, ez = hj.z - hi.z;
            if (ex * ex + ey * ey + ez * ez > d.bandHiColl) return;
            const float4 lj = __ldg(&d.posLo[j]);
            PairF q = pairDF(hj, lj, hi, li);
            if (!inBallDF(d, q.d2, R2, d.mgColl, P.distCollisionLimit2, i, j)) return;
            if (!sideOkDF(d, sc, hj, lj, q.d2, i, j)) return;
            float4 vhj = d.velHi[j], vlj = d.velLo[j];
            V3 dv = {diffDF(vh.x, vl.x, vhj.x, vlj.x), diffDF(vh.y, vl.y, vhj.y, vlj.y),
                     diffDF(vh.z, vl.z, vhj.z, vlj.z)};
            df fDT = dot3(dv, q.v);
            float rn = fabsf(q.v.x.h) + fabsf(q.v.y.h) + fabsf(q.v.z.h);
            float dn = fabsf(dv.x.h) + fabsf(dv.y.h) + fabsf(dv.z.h);
            float vjn = fabsf(vhj.x) + fabsf(vhj.y) + fabsf(vhj.z);
            float mg = 1e-9f * dn * rn + 1e-11f * (vin + vjn) * rn;
            bool pos;
            if (fDT.h > mg) pos = true;
            else if (fDT.h < -mg) pos = false;
            else {
                dvec4 pj = d.pos[j], vj = d.vel[j], vi = d.vel[i];
                PairG g = pairOf(pj, pi);
                pos = (vi.x - vj.x) * g.v0 + (vi.y - vj.y) * g.v1 + (vi.z - vj.z) * g.v2 > 0.0;
            }
            if (!pos) return;
            bool jf = d.type[j] == P.fluid;
            df rinv = rsqrtDF(q.d2);
            df k = fDT * (jf ? cF : cW) * (rinv * rinv);
            if (!jf) k = k * 2.0f;
            dvx -= q.v.x * k; dvy -= q.v.y * k; dvz -= q.v.z * k;
            any = true;
        });
    }
    d.dvel[i] = any ? make_dvec4(dD(dvx), dD(dvy), dD(dvz), 0.0) : make_dvec4(0, 0, 0, 0);
}
void launchCollisionDF(const Dev& d, cudaStream_t s) {
    launchVelDF(d, s);
    k_collision_df<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d);
    launchCollisionApply(d, s);
}

// ------------------------------------------------------------------ wall sweeps
struct MirrorDF {
    float4 mh, ml;
};
__device__ __forceinline__ MirrorDF mirrorDF(const Dev& d, dvec4 m) {
    MirrorDF o;
    splitPos(m, d.P, o.mh, o.ml);
    return o;
}
// MpsPndNeigh::calcWallNPCD, src/MpsPndNeigh.cpp:105-195
__global__ void __launch_bounds__(WALL_BLK) k_wall_npcd_df(Dev d) {
    __shared__ double sm[3][32];
    const MpsParams& P = d.P;
    const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
    forNearWall(d, [](int, int) {}, [&](int i, int g, int l) {
        const MirrorDF M = mirrorDF(d, d.mirror[i]);
        df sx = dfF(0.f), sy = dfF(0.f), sz = dfF(0.f);
        forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorS[i], l, [&](int j, int) {
            const PairF m = pairDF(__ldg(&d.posf[j]), __ldg(&d.posLo[j]), M.mh, M.ml);
            const df wS = weightDF(m.d2, RS, P.weightType).w;
            mac(sx, m.v.x, wS); mac(sy, m.v.y, wS); mac(sz, m.v.z, wS);
        });
        sx = laneSumDF<WALL_L>(sx); sy = laneSumDF<WALL_L>(sy); sz = laneSumDF<WALL_L>(sz);
        if (l == 0) { sm[0][g] = dD(sx); sm[1][g] = dD(sy); sm[2][g] = dD(sz); }
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
void launchWallNpcdDF(const Dev& d, cudaStream_t s) {
    if (d.P.wallType != 1) return;
    k_wall_npcd_df<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ correction matrix
// MpsVectorMatrix::correctionMatrix + inverseMatrix, src/MpsVectorMatrix.cpp:20-166: the
// moment matrix sum w/r^2 r r^T is accumulated in float-float and inverted through its
// adjugate in float-float (the reference eliminates without pivoting; both give the
// inverse to rounding), identity when det <= eps or numNeigh < 4.  The FP64 copy is the
// operator's output; the float-float copy feeds the DF32 pressure gradient.
__device__ __forceinline__ df recipDF(df a) {
    float y = 1.0f / a.h;
    df t = a * y;                              // ~1
    float e = fS(fS(1.0f, t.h), t.l);          // 1 - a y
    return quick2(y, fM(y, e));
}
__device__ __forceinline__ void corrFinish(const Dev& d, int i, int numNeigh, df m00, df m01, df m02, df m11,
                                           df m12, df m22, dvec4* c1, dvec4* c2, dvec4* c3, float2* cdf);
struct MomentsDF {
    df xx = {0.f, 0.f}, xy = {0.f, 0.f}, xz = {0.f, 0.f}, yy = {0.f, 0.f}, yz = {0.f, 0.f}, zz = {0.f, 0.f};
    __device__ __forceinline__ void add(const V3& v, df wr2) {
        const df t0 = v.x * wr2, t1 = v.y * wr2, t2 = v.z * wr2;
        mac(xx, t0, v.x); mac(xy, t0, v.y); mac(xz, t0, v.z);
        mac(yy, t1, v.y); mac(yz, t1, v.z); mac(zz, t2, v.z);
    }
    template <int L>
    __device__ __forceinline__ void sum() {
        xx = laneSumDF<L>(xx); xy = laneSumDF<L>(xy); xz = laneSumDF<L>(xz);
        yy = laneSumDF<L>(yy); yz = laneSumDF<L>(yz); zz = laneSumDF<L>(zz);
    }
};
template <int L>
__global__ void __launch_bounds__(BLK) k_corr_matrix_df(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    float4 hi = d.posf[i], li = d.posLo[i];
    const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
    MomentsDF M;
    forBitsOne(d.nbr + i, d.N0, laneShare<L>(d.maskS[i], l), [&](int j) { return loadPos(d, j); },
                 [&](int, int, const NbrPos& n) {
                     PairF q = pairDF(n.h, n.l, hi, li);
                     M.add(q.v, weightDF(q.d2, RS, P.weightType).wr2);
                 });
    M.sum<L>();
    if (l == 0) corrFinish(d, i, d.numNeigh[i], M.xx, M.xy, M.xz, M.yy, M.yz, M.zz, d.c1, d.c2, d.c3, d.corrDF);
}
// inverse of -coeffPressGrad * the moment matrix (identity when det <= eps or fewer than
// four neighbours), written as the FP64 rows and the float-float copy
__device__ __forceinline__ void corrFinish(const Dev& d, int i, int numNeigh, df m00, df m01, df m02, df m11,
                                           df m12, df m22, dvec4* c1, dvec4* c2, dvec4* c3, float2* cdf) {
    const MpsParams& P = d.P;
    const df c = K(d.k.negCPG);
    df A[9];
    A[0] = m00 * c; A[1] = m01 * c; A[2] = m02 * c;
    A[4] = m11 * c; A[5] = m12 * c; A[8] = m22 * c;
    A[3] = A[1]; A[6] = A[2]; A[7] = A[5];
    if (P.dim == 2) { A[2] = A[5] = A[6] = A[7] = dfF(0.f); A[8] = dfF(1.f); }
    df det = (A[0] * A[4] * A[8] + A[1] * A[5] * A[6] + A[2] * A[3] * A[7]) -
             (A[2] * A[4] * A[6] + A[1] * A[3] * A[8] + A[0] * A[5] * A[7]);
    df M[9];
    bool ident = numNeigh < 4 || !(det.h > (float)P.epsilonZero);
    if (ident) {
#pragma unroll
        for (int k = 0; k < 9; k++) M[k] = dfF((k % 4 == 0) ? 1.f : 0.f);
    } else {
        df r = recipDF(det);
        M[0] = (A[4] * A[8] - A[5] * A[7]) * r; M[1] = (A[2] * A[7] - A[1] * A[8]) * r;
        M[2] = (A[1] * A[5] - A[2] * A[4]) * r; M[3] = (A[5] * A[6] - A[3] * A[8]) * r;
        M[4] = (A[0] * A[8] - A[2] * A[6]) * r; M[5] = (A[2] * A[3] - A[0] * A[5]) * r;
        M[6] = (A[3] * A[7] - A[4] * A[6]) * r; M[7] = (A[1] * A[6] - A[0] * A[7]) * r;
        M[8] = (A[0] * A[4] - A[1] * A[3]) * r;
    }
#pragma unroll
    for (int k = 0; k < 9; k++) cdf[(size_t)k * d.N0 + i] = make_float2(M[k].h, M[k].l);
    c1[i] = make_dvec4(dD(M[0]), dD(M[1]), dD(M[2]), 0.0);
    c2[i] = make_dvec4(dD(M[3]), dD(M[4]), dD(M[5]), 0.0);
    c3[i] = make_dvec4(dD(M[6]), dD(M[7]), dD(M[8]), 0.0);
}
// float-float copy of matrices written through the field interface
__global__ void k_df_corr(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N0) return;
    dvec4 r[3] = {d.c1[i], d.c2[i], d.c3[i]};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        df x = dfD(r[a].x), y = dfD(r[a].y), z = dfD(r[a].z);
        d.corrDF[(size_t)(3 * a) * d.N0 + i] = make_float2(x.h, x.l);
        d.corrDF[(size_t)(3 * a + 1) * d.N0 + i] = make_float2(y.h, y.l);
        d.corrDF[(size_t)(3 * a + 2) * d.N0 + i] = make_float2(z.h, z.l);
    }
}
void launchCorrDF(const Dev& d, cudaStream_t s) { k_df_corr<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }
void launchCorrectionMatrixDF(const Dev& d, cudaStream_t s) {
#define LAUNCH(L) k_corr_matrix_df<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// ------------------------------------------------------------------ PND / NPCD
// MpsPndNeigh::calcPndnNeighNPCD, src/MpsPndNeigh.cpp:199-331
// CORR: the correction matrix's moment sums over the reS entries in the same pass (one
// pair evaluation serves both; the PND sums take the entries also inside reL, in the same
// ascending order as the plain sweep, so both results equal the separate kernels').
template <bool CORR, int L>
__global__ void __launch_bounds__(BLK, 9) k_pnd_npcd_df(Dev d, bool bc) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    float4 hi = d.posf[i], li = d.posLo[i];
    const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
    const Mask mL = d.maskL[i], mS = d.maskS[i];
    df ni = dfF(0.f), nx = ni, ny = ni, nz = ni;
    MomentsDF M;
    forBitsOne(d.nbr + i, d.N0, laneShare<L>(CORR ? mS : (mL & mS), l), [&](int j) { return loadPos(d, j); },
                 [&](int, int k, const NbrPos& n) {
                     PairF q = pairDF(n.h, n.l, hi, li);
                     WeightDF w = weightDF(q.d2, RS, P.weightType);
                     if (CORR) M.add(q.v, w.wr2);
                     if (!CORR || maskHas(mL, k)) {
                         acc(ni, w.w);
                         mac(nx, q.v.x, w.w); mac(ny, q.v.y, w.w); mac(nz, q.v.z, w.w);
                     }
                 });
    ni = laneSumDF<L>(ni); nx = laneSumDF<L>(nx); ny = laneSumDF<L>(ny); nz = laneSumDF<L>(nz);
    if (CORR) M.sum<L>();
    if (l != 0) return;
    const int nn = d.nNeighWall[i] + maskCount(mL);
    double nd = dD(ni);
    dvec4 np = d.npcd[i];
    np.x += dD(nx); np.y += dD(ny); np.z += dD(nz);
    if (P.pndType == 0 || P.pndType == 1) {
        d.pndki[i] = d.pndi[i];
        d.pndi[i] = nd + d.pndWall[i];
    }
    double pndSmall = nd + d.pndWall[i];
    d.pndSmall[i] = pndSmall;
    d.numNeigh[i] = nn;
    if (nd > P.epsilonZero) { np.x /= pndSmall; np.y /= pndSmall; np.z /= pndSmall; }
    d.npcd[i] = np;
    d.npcd2[i] = np.x * np.x + np.y * np.y + np.z * np.z;
    dvec4 nw = d.polyNormal[i];
    d.devDot[i] = (np.x * nw.x + np.y * nw.y + np.z * nw.z < 0.0) ? 1.0 : -1.0;
    if (bc) d.bc[i] = boundaryCondition(d, i, pndSmall, nn, np.x * np.x + np.y * np.y + np.z * np.z);
    // into the staging arrays: the correction-matrix operator publishes them (the reference
    // writes the matrix there, not in this sweep)
    if (CORR) corrFinish(d, i, nn, M.xx, M.xy, M.xz, M.yy, M.yz, M.zz, d.c1n, d.c2n, d.c3n, d.corrDFn);
}
void launchPndNeighNpcdDF(const Dev& d, cudaStream_t s, bool withCorrection, bool withBC) {
#define LAUNCH(L)                                                                            \
    if (withCorrection) k_pnd_npcd_df<true, L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d, withBC);    \
    else k_pnd_npcd_df<false, L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d, withBC)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// ------------------------------------------------------------------ PPE assembly
// MpsPressure::solvePressurePoissonPnd, src/MpsPressure.cpp:169-286 (matrix values are
// assembled in float-float and stored in FP64)
template <int L>
__global__ void __launch_bounds__(128, 9) k_ppe_assemble_df(Dev d, PpeBuffers B) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (l == 0) B.x[i] = d.pressPPE[i];   // the start of a solve from the previous solution
    int bci = d.bc[i];
    if (bci == P.other || bci == P.surface) {
        if (l == 0) {
            B.diag[i] = 1.0; B.diagf[i] = 1.0f; B.diagInvf[i] = 1.0f; B.rowLen[i] = 0; B.b[i] = 0.0;
            B.mfMask[i] = maskNone();
        }
        warpCount(d.counters + 1, 0u);
        return;
    }
    float4 hi = d.posf[i], li = d.posLo[i];
    const RadiusDF RL = {K(d.k.reL), K(d.k.invReL)};
    const df cP = K(d.k.cPPE);
    df sum = dfF(0.f), src = dfF(0.f);
    const Mask mL = d.maskL[i];
    const int* row = d.nbr + i;
    const size_t base = ellBase(B, i);
    int len = 0;
    Mask mm = maskNone();
    if (L > 1) {   // the matrix entries of the whole row first: an entry's place is its rank
        forMaskLane<L>(d, i, mL, l, [&](int j, size_t, int k) {
            if (d.type[j] != P.dummyWall && d.bc[j] == P.inner) maskSet(mm, k);
        });
        mm = laneOr<L>(mm);
        len = maskCount(mm);
    }
    struct Nbr { NbrPos p; int type, bc; };
    forBitsTwo(row, d.N0, laneShare<L>(mL, l),
                 [&](int j) { return Nbr{loadPos(d, j), __ldg(&d.type[j]), __ldg(&d.bc[j])}; },
                 [&](int j, int k, const Nbr& n) {
                     PairF q = pairDF(n.p.h, n.p.l, hi, li);
                     df wL = weightDF(q.d2, RL, P.weightType).w;
                     if (n.type == P.dummyWall) {
                         src -= (q.v.x * K(d.k.g[0]) + q.v.y * K(d.k.g[1]) + q.v.z * K(d.k.g[2])) * wL * K(d.k.cPPEg);
                         return;
                     }
                     df mij = wL * cP;
                     acc(sum, -mij);
                     if (n.bc != P.inner) return;
                     int at;
                     if (L > 1) at = maskRank(mm, k);
                     else { at = len++; maskSet(mm, k); }
                     const size_t e = base + (size_t)at * B.ellStride;
                     B.val[e] = dD(mij);
                     B.valf[e] = mij.h;   // the FP32 copy of the mixed solver (hi part = fl32)
                     B.col[e] = j;
                 });
    sum = laneSumDF<L>(sum);
    src = laneSumDF<L>(src);
    if (l == 0) {
        B.mfMask[i] = mm;
        double rho = P.DNS_FL1;
        double dg = dD(sum) - P.alphaCompressibility * rho / (P.timeStep * P.timeStep);
        B.diag[i] = dg;
        B.diagf[i] = (float)dg;
        B.diagInvf[i] = 1.0f / (float)dg;
        B.rowLen[i] = len;
        B.b[i] = dD(src) + ppeSource(d, i, rho);
    }
    warpCount(d.counters + 1, l == 0 ? (unsigned)len : 0u);
}
void launchPpeAssembleDF(const Dev& d, const PpeBuffers& B, cudaStream_t s) {
    cudaMemsetAsync(d.counters + 1, 0, sizeof(unsigned long long), s);
#define LAUNCH(L) k_ppe_assemble_df<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d, B)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// ------------------------------------------------------------------ pressure gradient
// MpsPressure::calcPressGradient, src/MpsPressure.cpp:1217-1338
template <int L>
__global__ void __launch_bounds__(BLK, 8) k_press_grad_df(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    float4 hi = d.posf[i], li = d.posLo[i];
    const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
    df Pi = loadDF(d.pressDF, i), pmin = Pi;
    double ni = d.pndi[i];
    int gt = P.gradientType;
    const Mask mS = laneShare<L>(d.maskS[i], l);
    const int* row = d.nbr + i;
    if (gt == 0 || gt == 2) {
        forBitsTwo(row, d.N0, mS, [&](int j) { return __ldg(d.pressDF + j); }, [&](int, int, float2 p) {
            const df pj = {p.x, p.y};
            if (pmin > pj) pmin = pj;
        });
#pragma unroll
        for (int o = 1; o < L; o <<= 1) {
            const df q = {__shfl_xor_sync(laneGroup<L>(), pmin.h, o), __shfl_xor_sync(laneGroup<L>(), pmin.l, o)};
            if (pmin > q) pmin = q;
        }
        if (l == 0) ((float2*)d.pAux)[i] = make_float2(pmin.h, pmin.l);   // for the wall term
    }
    df base = (gt == 0) ? -pmin : (gt == 1 ? Pi : Pi - pmin - pmin);
    // sum of r_ij f_ij; with gradient correction C (constant per particle) is applied to
    // the sum once: sum (C r) f = C (sum r f)
    df ax = dfF(0.f), ay = ax, az = ax;
    struct Nbr { NbrPos p; float2 pr; };
    forBitsTwo(row, d.N0, mS, [&](int j) { return Nbr{loadPos(d, j), __ldg(d.pressDF + j)}; },
                 [&](int j, int, const Nbr& n) {
                     PairF q = pairDF(n.p.h, n.p.l, hi, li);
                     WeightDF w = weightDF(q.d2, RS, P.weightType);
                     df f;
                     if (gt <= 2) f = (df{n.pr.x, n.pr.y} + base) * w.wr2;
                     else {
                         double nj = d.pndi[j], Pj = d.press[j], Pid = d.press[i];
                         f = (ni > P.epsilonZero && nj > P.epsilonZero) ? dfD(ni * Pj / nj + nj * Pid / ni) * w.wr2 : w.w;
                     }
                     mac(ax, q.v.x, f); mac(ay, q.v.y, f); mac(az, q.v.z, f);
                 });
    ax = laneSumDF<L>(ax); ay = laneSumDF<L>(ay); az = laneSumDF<L>(az);
    if (l != 0) return;
    if (P.gradientCorrection) {
        df C[9];
#pragma unroll
        for (int k = 0; k < 9; k++) C[k] = loadDF(d.corrDF + (size_t)k * d.N0, i);
        df bx = C[0] * ax + C[1] * ay + C[2] * az;
        df by = C[3] * ax + C[4] * ay + C[5] * az;
        df bz = C[6] * ax + C[7] * ay + C[8] * az;
        ax = bx; ay = by; az = bz;
    }
    d.acc[i] = make_dvec4(dD(ax) * d.cPG, dD(ay) * d.cPG, dD(az) * d.cPG, 0.0);
}
void launchPressGradientDF(const Dev& d, cudaStream_t s) {
    launchPressDF(d, s);
#define LAUNCH(L) k_press_grad_df<L><<<gridFor(d.N0 * L, BLK), BLK, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// MpsPressure::calcWallPressGradient + repulsive forces, src/MpsPressure.cpp:1341-1611
__global__ void __launch_bounds__(WALL_BLK) k_wall_press_grad_df(Dev d, bool fresh) {
    __shared__ double sm[3][32], pmn[32];
    const MpsParams& P = d.P;
    const int gt = P.gradientType;
    const double vm = fmin(*d.velMax, P.expectMaxVelocity);
    const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
    forNearWall(d, [](int, int) {}, [&](int i, int g, int l) {
        const MirrorDF M = mirrorDF(d, d.mirror[i]);
        const double Pid = d.press[i], ni = d.pndi[i];
        const df Pi = loadDF(d.pressDF, i);
        df pmin = Pi;
        if ((gt == 0 || gt == 2) && fresh) pmin = loadDF((const float2*)d.pAux, i);
        else if (gt == 0 || gt == 2) {
            forMaskLane<WALL_L>(d, i, d.maskS[i], l, [&](int j, size_t, int) {
                const df pj = loadDF(d.pressDF, j);
                if (pmin > pj) pmin = pj;
            });
#pragma unroll
            for (int o = 1; o < WALL_L; o <<= 1) {
                const df q = {__shfl_xor_sync(laneGroup<WALL_L>(), pmin.h, o), __shfl_xor_sync(laneGroup<WALL_L>(), pmin.l, o)};
                if (pmin > q) pmin = q;
            }
        }
        const df base = (gt == 0) ? -pmin : (gt == 1 ? Pi : Pi - pmin - pmin);
        df sx = dfF(0.f), sy = sx, sz = sx;
        forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorS[i], l, [&](int j, int) {
            const PairF m = pairDF(__ldg(&d.posf[j]), __ldg(&d.posLo[j]), M.mh, M.ml);
            const WeightDF w = weightDF(m.d2, RS, P.weightType);
            df f;
            if (gt <= 2) f = (loadDF(d.pressDF, j) + base) * w.wr2;
            else {
                double nj = d.pndi[j], Pj = d.press[j];
                f = (ni > P.epsilonZero && nj > P.epsilonZero) ? dfD(ni * Pj / nj + nj * Pid / ni) * w.wr2 : w.w;
            }
            mac(sx, m.v.x, f); mac(sy, m.v.y, f); mac(sz, m.v.z, f);
        });
        sx = laneSumDF<WALL_L>(sx); sy = laneSumDF<WALL_L>(sy); sz = laneSumDF<WALL_L>(sz);
        if (l == 0) { sm[0][g] = dD(sx); sm[1][g] = dD(sy); sm[2][g] = dD(sz); pmn[g] = dD(pmin); }
    }, [&](int i, int g) {
        const dvec4 pi = d.pos[i], mi = d.mirror[i];
        const double Pid = d.press[i], ni = d.pndi[i], pmind = pmn[g];
        const ReflG r = makeRefl(pi, mi, P.epsilonZero, true);
        double ax = sm[0][g], ay = sm[1][g], az = sm[2][g];
        PairM s = pairMirror(pi, mi);
        if (s.dm2 < P.reS2) {
            double wS = wfun(sqrt(s.dm2), P.reS, P.weightType);
            if (gt == 0) wS = wS * ((Pid - pmind) / s.dm2);
            else if (gt == 1) wS = wS * ((Pid + Pid) / s.dm2);
            else if (gt == 2) wS = wS * ((Pid + Pid - 2.0 * pmind) / s.dm2);
            else if (gt == 3 && ni > P.epsilonZero) wS = wS * ((ni * Pid / ni + ni * Pid / ni) / s.dm2);
            ax += s.m0 * wS; ay += s.m1 * wS; az += s.m2 * wS;
        }
        double f[3];
        wallRepulsion(P, r, vm * vm, f);
        double gr[3];
#pragma unroll
        for (int a = 0; a < 3; a++)
            gr[a] = P.relaxPress * (r.R[3 * a] * ax + r.R[3 * a + 1] * ay + r.R[3 * a + 2] * az) * P.coeffPressGrad - f[a];
        dvec4 a = d.acc[i];
        a.x += gr[0] / P.DNS_FL1; a.y += gr[1] / P.DNS_FL1; a.z += gr[2] / P.DNS_FL1;
        d.acc[i] = a;
        double vf = (P.dim == 3) ? P.partDist * P.partDist * P.partDist : P.partDist * P.partDist;
        dvec4 fw = d.forceWall[i];
        fw.x += -gr[0] * vf; fw.y += -gr[1] * vf; fw.z += -gr[2] * vf;
        d.forceWall[i] = fw;
    });
}
void launchWallPressGradientDF(const Dev& d, cudaStream_t s, bool fresh) {
    if (d.P.wallType != 1) return;
    if (!fresh) launchPressDF(d, s);
    k_wall_press_grad_df<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d, fresh);
}

// ------------------------------------------------------------------ wall viscosity
// MpsViscosity::calcWallNoSlipViscosity / calcWallSlipViscosity, src/MpsViscosity.cpp:1527-1910
__global__ void __launch_bounds__(WALL_BLK) k_wall_visc_df(Dev d) {
    __shared__ double sm[3][32], vm[3][32];
    const MpsParams& P = d.P;
    const bool noslip = P.slipCondition == 0;
    const double mu = P.KNM_VS1 * P.DNS_FL1;
    const df neuF = K(d.k.neuWall);
    const RadiusDF RL = {K(d.k.reL), K(d.k.invReL)};
    auto matrix = [&](int i, double M[9]) {
        if (noslip) {
#pragma unroll
            for (int k = 0; k < 9; k++) M[k] = (k % 4 == 0) ? -1.0 : 0.0;
            return;
        }
        const ReflG r = makeRefl(d.pos[i], d.mirror[i], P.epsilonZero, false);
#pragma unroll
        for (int k = 0; k < 9; k++) M[k] = r.R[k];
    };
    forNearWall(d, [&](int i, int g) {
        const dvec4 vi = d.vel[i];
        double M[9];
        matrix(i, M);
#pragma unroll
        for (int a = 0; a < 3; a++) vm[a][g] = M[3 * a] * vi.x + M[3 * a + 1] * vi.y + M[3 * a + 2] * vi.z;
    }, [&](int i, int g, int l) {
        const MirrorDF Mi = mirrorDF(d, d.mirror[i]);
        const df vmx = dfD(vm[0][g]), vmy = dfD(vm[1][g]), vmz = dfD(vm[2][g]);
        df sx = dfF(0.f), sy = sx, sz = sx;
        forBitsShared<WALL_L>(d.nbr + i, d.N0, d.mirrorL[i], l, [&](int j, int) {
            const PairF m = pairDF(__ldg(&d.posf[j]), __ldg(&d.posLo[j]), Mi.mh, Mi.ml);
            const df c = weightDF(m.d2, RL, P.weightType).w * neuF;
            float4 vhj = d.velHi[j], vlj = d.velLo[j];
            mac(sx, dfOf(vhj.x, vlj.x) - vmx, c);
            mac(sy, dfOf(vhj.y, vlj.y) - vmy, c);
            mac(sz, dfOf(vhj.z, vlj.z) - vmz, c);
        });
        sx = laneSumDF<WALL_L>(sx); sy = laneSumDF<WALL_L>(sy); sz = laneSumDF<WALL_L>(sz);
        if (l == 0) { sm[0][g] = dD(sx); sm[1][g] = dD(sy); sm[2][g] = dD(sz); }
    }, [&](int i, int g) {
        const dvec4 pi = d.pos[i], vi = d.vel[i], mi = d.mirror[i];
        double M[9];
        matrix(i, M);
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
void launchWallViscosityDF(const Dev& d, cudaStream_t s) {
    if (d.P.wallType != 1) return;
    launchVelDF(d, s);
    k_wall_visc_df<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d);
}

// ------------------------------------------------------------------ shifting
// MpsShifting (src/MpsShifting.cpp:23-101 type 1, :432-691 type 2) at the post-corrector
// positions through the 27 buckets.  Each sweep runs in bucket order over the listed
// particles and once more over the unlisted ones; entries are the reS ball minus the
// mirror side, decided exactly as in the FP64 tier.
template <class Op, bool STRAY>
__global__ void __launch_bounds__(BLK) k_shift_scan_df(Dev d, Op op) {
    const int i = scanParticle<STRAY>(d);
    if (i < 0) return;
    typename Op::State st;
    const bool on = op.begin(d, i, st);
    if (on) {
        const MpsParams& P = d.P;
        const dvec4 pi = d.pos[i];
        const float4 hi = d.posf[i], li = d.posLo[i];
        const SideDF sc = sideDF(d, i, pi);
        const df R2 = K(d.k.reS2);
        forCellsDF(d, pi, hi, d.bandHiS, [&](int j, int s, float4 hj) {
            if (j == i) return;
            const float4 lj = __ldg(&d.posLoCell[s]);
            PairF q = pairDF(hj, lj, hi, li);
            if (!inBallDF(d, q.d2, R2, d.mgS, P.reS2, i, j)) return;
            if (!sideOkDF(d, sc, hj, lj, q.d2, i, j)) return;
            op.visit(d, st, j, q);
        });
    }
    op.end(d, i, st, on);
}
template <class Op>
static void launchShiftScanDF(const Dev& d, const Op& op, cudaStream_t s) {
    k_shift_scan_df<Op, false><<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, op);
    k_shift_scan_df<Op, true><<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, op);
}

// dw/dr of MpsParticle::delWeight (src/MpsParticle.cpp) from r^2, float-float
__device__ __forceinline__ df dweightDF(df d2, const RadiusDF& R, int t) {
    df rinv = rsqrtDF(d2);
    switch (t) {
        case 1: return -(R.re * (rinv * rinv)) + R.invRe;
        case 2: return -(R.re * (rinv * rinv)) - R.invRe;
        case 3: { df a = -(d2 * rinv * R.invRe) + 1.0f; return (a * a) * (R.invRe * -3.0f); }
        case 4: { df a = -(d2 * rinv * R.invRe) + 1.0f; return a * (R.invRe * -2.0f); }
        default: return -(R.re * (rinv * rinv));
    }
}

// type 1: dv_i = sum dw(r_ij) (v_j - v_i) over fluid particles, applied to inner ones
struct ShiftVelDF {
    struct State { float4 vh, vl; df ux, uy, uz; };
    __device__ bool begin(const Dev& d, int i, State& st) const {
        st.vh = d.velHi[i]; st.vl = d.velLo[i];
        st.ux = st.uy = st.uz = dfF(0.f);
        return d.type[i] == d.P.fluid;
    }
    __device__ void visit(const Dev& d, State& st, int j, const PairF& q) const {
        const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
        df dw = dweightDF(q.d2, RS, d.P.weightType);
        float4 vhj = d.velHi[j], vlj = d.velLo[j];
        mac(st.ux, diffDF(vhj.x, vlj.x, st.vh.x, st.vl.x), dw);
        mac(st.uy, diffDF(vhj.y, vlj.y, st.vh.y, st.vl.y), dw);
        mac(st.uz, diffDF(vhj.z, vlj.z, st.vh.z, st.vl.z), dw);
    }
    __device__ void end(const Dev& d, int i, State& st, bool on) const {
        bool apply = on && d.bc[i] == d.P.inner;
        d.shift[i] = apply ? make_dvec4(dD(st.ux), dD(st.uy), dD(st.uz), 0.0) : make_dvec4(0, 0, 0, 0);
    }
};
// type 2, concentration: C_i = (sum w(r_ij) + wall PND) / pndSmallZero, every particle
struct ConcDF {
    struct State { df sum; };
    __device__ bool begin(const Dev&, int, State& st) const { st.sum = dfF(0.f); return true; }
    __device__ void visit(const Dev& d, State& st, int, const PairF& q) const {
        const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
        acc(st.sum, weightDF(q.d2, RS, d.P.weightType).w);
    }
    __device__ void end(const Dev& d, int i, State& st, bool) const {
        d.conc[i] = (dD(st.sum) + d.pndWall[i]) / d.P.pndSmallZero;
    }
};
__global__ void k_df_conc(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N0) return;
    df c = dfD(d.conc[i]);
    d.concDF[i] = make_float2(c.h, c.l);
}
// type 2, gradient: grad C_i = -coeffPressGrad sum (C_i + C_j) w/r^2 r_ij over fluid
// particles; the shift of inner particles is -coeffShifting2 grad C_i
struct GradConcDF {
    struct State { df ci, gx, gy, gz; };
    __device__ bool begin(const Dev& d, int i, State& st) const {
        st.ci = loadDF(d.concDF, i);
        st.gx = st.gy = st.gz = dfF(0.f);
        return d.type[i] == d.P.fluid;
    }
    __device__ void visit(const Dev& d, State& st, int j, const PairF& q) const {
        const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
        df cc = (st.ci + loadDF(d.concDF, j)) * weightDF(q.d2, RS, d.P.weightType).wr2;
        mac(st.gx, q.v.x, cc); mac(st.gy, q.v.y, cc); mac(st.gz, q.v.z, cc);
    }
    __device__ void end(const Dev& d, int i, State& st, bool on) const {
        const MpsParams& P = d.P;
        dvec4 sh = make_dvec4(0, 0, 0, 0);
        if (on) {
            double gx = dD(st.gx) * -P.coeffPressGrad, gy = dD(st.gy) * -P.coeffPressGrad,
                   gz = dD(st.gz) * -P.coeffPressGrad;
            d.gradC[i] = make_dvec4(gx, gy, gz, 0.0);
            if (d.bc[i] == P.inner)
                sh = make_dvec4(-P.coeffShifting2 * gx, -P.coeffShifting2 * gy, -P.coeffShifting2 * gz, 0.0);
        }
        d.shift[i] = sh;
    }
};
// type 2, wall contribution (src/MpsShifting.cpp:578-691) at the shifted positions:
// mirror entries of near-wall fluid particles, reflected by the wall plane of i.
__global__ void __launch_bounds__(WALL_BLK) k_wall_grad_conc_df(Dev d, bool skin) {
    __shared__ WallCand W;
    __shared__ double sm[3][32];
    const MpsParams& P = d.P;
    const RadiusDF RS = {K(d.k.reS), K(d.k.invReS)};
    const int nn = *d.nearCount;
    const bool useSkin = skin && !*(volatile int*)d.skinFlag;
    for (int base = blockIdx.x * 32; base < nn; base += gridDim.x * 32) {
        wallCandidates(d, W, base, nn, useSkin);
        __syncthreads();
        const int g = threadIdx.x / WALL_L, l = threadIdx.x & (WALL_L - 1);
        if (base + g < nn) {
            const int i = d.nearList[base + g];
            const MirrorDF M = mirrorDF(d, d.mirror[i]);
            const df ci = loadDF(d.concDF, i);
            df sx = dfF(0.f), sy = sx, sz = sx;
            forWallCand(d, W, i, g, l, [&](int j) {
                const PairF m = pairDF(__ldg(&d.posf[j]), __ldg(&d.posLo[j]), M.mh, M.ml);
                const df cc = (ci + loadDF(d.concDF, j)) * weightDF(m.d2, RS, P.weightType).wr2;
                mac(sx, m.v.x, cc); mac(sy, m.v.y, cc); mac(sz, m.v.z, cc);
            });
            sx = laneSumDF<WALL_L>(sx); sy = laneSumDF<WALL_L>(sy); sz = laneSumDF<WALL_L>(sz);
            if (l == 0) { sm[0][g] = dD(sx); sm[1][g] = dD(sy); sm[2][g] = dD(sz); }
        }
        __syncthreads();
        if (threadIdx.x < 32 && base + (int)threadIdx.x < nn)
            wallGradConcEnd(d, d.nearList[base + threadIdx.x], sm[0][threadIdx.x], sm[1][threadIdx.x], sm[2][threadIdx.x]);
        __syncthreads();
    }
}
static void launchWallGradConcDF(const Dev& d, cudaStream_t s, bool list) {
    if (list) launchSkinCheck(d, s, false);
    else launchNearList(d, s);
    k_wall_grad_conc_df<<<wallGrid(d.N0), WALL_BLK, 0, s>>>(d, list);
    launchApplyShiftNear(d, s);
}
// The shifting sums over the list of the post-corrector positions (filtered from the skin
// list) instead of the 27-bucket scan: the reS-ball entries off the mirror side are the
// maskS entries of that list, in scan order, so the sums are those of k_shift_scan_df.
template <class Op>
__global__ void __launch_bounds__(BLK) k_shift_list_df(Dev d, Op op) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    typename Op::State st;
    const bool on = op.begin(d, i, st);
    if (on) {
        const float4 hi = d.posf[i], li = d.posLo[i];
        forBitsTwo(d.nbr + i, d.N0, d.maskS[i], [&](int j) { return loadPos(d, j); },
                     [&](int j, int, const NbrPos& n) { op.visit(d, st, j, pairDF(n.h, n.l, hi, li)); });
    }
    op.end(d, i, st, on);
}
// Shifting from the list of the current positions (built by the caller: filter + masks).
void launchShiftingListDF(const Dev& d, cudaStream_t s) {
    const MpsParams& P = d.P;
    if (P.shiftingType == 1) {
        launchVelDF(d, s);
        k_shift_list_df<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, ShiftVelDF());
        launchShiftVelApply(d, s);
        return;
    }
    k_shift_list_df<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, ConcDF());
    k_df_conc<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    k_shift_list_df<<<gridFor(d.N0, BLK), BLK, 0, s>>>(d, GradConcDF());
    launchApplyShift(d, s);
    if (P.wallType == 1) launchWallGradConcDF(d, s, true);
}
void launchShiftingDF(const Dev& d, cudaStream_t s) {
    const MpsParams& P = d.P;
    if (P.shiftingType != 1 && P.shiftingType != 2) return;
    launchPosf(d, s);   // post-corrector positions (hi/lo, particle and bucket order)
    if (P.shiftingType == 1) {
        launchVelDF(d, s);
        launchShiftScanDF(d, ShiftVelDF(), s);
        launchShiftVelApply(d, s);
        return;
    }
    launchShiftScanDF(d, ConcDF(), s);
    k_df_conc<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    launchShiftScanDF(d, GradConcDF(), s);
    launchApplyShift(d, s);
    if (P.wallType == 1) launchWallGradConcDF(d, s, false);
}

// ------------------------------------------------------------------ start-of-step list
// Viscosity over the start-of-step list instead of the 27 buckets (k_visc_df's entries, in the
// scan order within a lane), L lanes per particle: the FP32 copies decide the 56 entries of a
// row first (mps_lanes.cuh), the float-float sums walk the 32 inside (559 -> 369 us at 864k
// particles).
template <int L>
__global__ void __launch_bounds__(128) k_visc_list_df(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const float4 hi = d.posf[i], li = d.posLo[i];
    const float4 vh = d.velHi[i], vl = d.velLo[i];
    const RadiusDF RL = {K(d.k.reL), K(d.k.invReL)};
    df ax = dfF(0.f), ay = dfF(0.f), az = dfF(0.f);
    struct Nbr { NbrPos p; float4 vh, vl; int type; };
    auto load = [&](int j) { return Nbr{loadPos(d, j), __ldg(&d.velHi[j]), __ldg(&d.velLo[j]), __ldg(&d.type[j])}; };
    auto add = [&](int, int, const Nbr& n) {
        const PairF q = pairDF(n.p.h, n.p.l, hi, li);
        const df c = weightDF(q.d2, RL, P.weightType).w * (n.type == P.wall ? K(d.k.neuW) : K(d.k.neuF));
        mac(ax, diffDF(n.vh.x, n.vl.x, vh.x, vl.x), c);
        mac(ay, diffDF(n.vh.y, n.vl.y, vh.y, vl.y), c);
        mac(az, diffDF(n.vh.z, n.vl.z, vh.z, vl.z), c);
    };
    const int c = d.nbrCount[i];
    if (c <= d.K) {
        const int* row = d.nbr + i;
        const SideF sd = sideF(d, i, d.pos[i]);
        const Mask m = rowMask<L>(d, row, l, c, [&](int j, float4 hj) {
            const float d2f = dist2f(hj, hi);
            return insideF(d, d2f, d.bandLoL, d.bandHiL, P.reL2, i, j) && sideOKF(d, sd, hj, d2f, i, j);
        });
        forBitsTwo(row, d.N0, m, load, add);
    } else if (l == 0) {   // the row overflowed: scan the buckets
        const dvec4 pi = d.pos[i];
        const SideDF sc = sideDF(d, i, pi);
        const df R2 = K(d.k.reL2);
        forCellsDF(d, pi, hi, d.bandHiL, [&](int j, int s, float4 hj) {
            if (j == i) return;
            const float4 lj = __ldg(&d.posLoCell[s]);
            const df d2 = pairDF(hj, lj, hi, li).d2;
            if (inBallDF(d, d2, R2, d.mgL, P.reL2, i, j) && sideOkDF(d, sc, hj, lj, d2, i, j)) add(j, 0, load(j));
        });
    }
    ax = laneSumDF<L>(ax); ay = laneSumDF<L>(ay); az = laneSumDF<L>(az);
    const double cv = P.coeffViscMultiphase;
    if (l == 0) d.acc[i] = make_dvec4(cv * dD(ax), cv * dD(ay), cv * dD(az), 0.0);
}
void launchViscosityListDF(const Dev& d, cudaStream_t s) {
    launchVelDF(d, s);
#define LAUNCH(L) k_visc_list_df<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// The skin list covers the list of the current positions while every particle is within
// half the skin of its start position (FP32 test with margin).
__global__ void k_skin_check(Dev d, bool clear) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (clear && i == 0) { *d.rescan = 0; d.counters[0] = 0ull; }
    if (i >= liveN(d)) return;
    float4 a = d.posf[i], b = d.posSkin[i];
    float ex = a.x - b.x, ey = a.y - b.y, ez = a.z - b.z;
    if (!(ex * ex + ey * ey + ez * ez <= d.skinMove2)) d.skinFlag[0] = 1;
}
void launchSkinCheck(const Dev& d, cudaStream_t s, bool clear) {
    k_skin_check<<<gridFor(d.N0, 256), 256, 0, s>>>(d, clear);
}
