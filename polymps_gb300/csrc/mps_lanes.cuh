// mps_lanes.cuh — L lanes of a warp per particle for the neighbour sweeps, and the FP32 tests
// that settle most of a sweep's decisions before any FP64 operation.
//
// GB300 issues FP64 at 1/64 of the FP32 rate, so an FP64 sweep is bound by the FP64
// operations its warps issue, whether one lane or all 32 need them.  The sweeps therefore run
// in two phases: the FP32 copies decide each row entry (an entry inside the rounding band of
// a decision takes the reference's FP64 expression, out of line) and leave a bit mask; then
// the FP64 sums walk the set bits, so the lanes of a warp stay in step through them.
#pragma once
#include "mps_df.cuh"

// Lanes per particle for n particles.  From 40k particles on the sweeps are bound by the FP64
// pipe and one lane per particle keeps its lanes busiest; below, the chip is not full and a
// row's chain of gathers and FP64 sums is the time of the sweep, which L lanes shorten.  The
// viscosity sweep with 1, 4 and 8 lanes: 6.9k particles 64 / 28 / 22 us, 18.5k 63 / 44 / 51 us,
// 32k 74 / 68 / 77 us, 55k 94 / 110 / 122 us, 108k 166 / 200 / 231 us.
static inline int lanesFor(int n) { return n >= 40000 ? 1 : (n >= 12000 ? 4 : 8); }
// Launch a kernel template over its lane count: KERNEL(L) expands to the launch for L lanes.
#define MPS_FOR_LANES(n, KERNEL)                                                                  \
    do {                                                                                          \
        switch (lanesFor(n)) {                                                                    \
            case 1: KERNEL(1); break;                                                             \
            case 4: KERNEL(4); break;                                                             \
            default: KERNEL(8); break;                                                            \
        }                                                                                         \
    } while (0)

// Row and lane of the calling thread; the lanes of a row are neighbours within one warp.
template <int L>
__device__ __forceinline__ int laneRow() { return (int)((blockIdx.x * blockDim.x + threadIdx.x) / L); }
template <int L>
__device__ __forceinline__ int laneOf() { return (int)(threadIdx.x & (L - 1)); }
template <int L>
__device__ __forceinline__ unsigned laneGroup() {
    return L == 1 ? 1u << (threadIdx.x & 31) : ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
}
// Sums over the lanes of a row: every lane of the group gets the same bits (a symmetric tree).
template <int L>
__device__ __forceinline__ double laneSum(double v) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(laneGroup<L>(), v, o);
    return v;
}
template <int L>
__device__ __forceinline__ int laneSum(int v) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(laneGroup<L>(), v, o);
    return v;
}
template <int L>
__device__ __forceinline__ Mask laneOr(Mask m) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
        m.lo |= __shfl_xor_sync(laneGroup<L>(), m.lo, o);
        m.hi |= __shfl_xor_sync(laneGroup<L>(), m.hi, o);
    }
    return m;
}
// The entries of a mask that lane l takes: k with k mod L == l.
template <int L>
__device__ __forceinline__ Mask laneShare(Mask m, int l) {
    if (L == 1) return m;
    static_assert(L == 1 || L == 4 || L == 8, "the lane counts of lanesFor");
    const unsigned long long p = (L == 4 ? 0x1111111111111111ull : 0x0101010101010101ull) << l;
    m.lo &= p; m.hi &= p;
    return m;
}
// Set bits below bit k.
__device__ __forceinline__ int maskRank(const Mask& m, int k) {
    if (k < 64) return __popcll(m.lo & ((1ull << k) - 1ull));
    return __popcll(m.lo) + __popcll(m.hi & ((1ull << (k - 64)) - 1ull));
}

// The reference's FP64 decisions, out of line: inlined, the compiler predicates them into every
// entry and their FP64 operations then run for all of them.
static __device__ __noinline__ bool pairInsideExact(const dvec4* pos, int j, int i, double R2) {
    return pairOf(pos[j], pos[i]).d2 < R2;
}
static __device__ __noinline__ bool mirrorInsideExact(const dvec4* pos, const dvec4* mirror, int j, int i, double R2) {
    return pairMirror(pos[j], mirror[i]).dm2 < R2;
}
static __device__ __noinline__ bool pairSideExact(const dvec4* pos, const dvec4* mirror, int j, int i) {
    const dvec4 pj = pos[j];
    return pairOf(pj, pos[i]).d2 < pairMirror(pj, mirror[i]).dm2;
}

// Minimum as `if (m > x) m = x` by integer comparisons of the ordered bits (a NaN x or m
// leaves m, as in FP64).
__device__ __forceinline__ long long orderedBits(double x) {
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ bool nanBits(double x) {
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ void minBits(double& m, double x) {
    if (orderedBits(m) > orderedBits(x) && !nanBits(x) && !nanBits(m)) m = x;
}

// FP32 squared distance of two position copies
__device__ __forceinline__ float dist2f(float4 a, float4 b) {
    const float ex = a.x - b.x, ey = a.y - b.y, ez = a.z - b.z;
    return ex * ex + ey * ey + ez * ez;
}
// The mirror-side test of particle i (SideCtx) with the mirror's FP32 copy: |x_j - x_i|^2 and
// |x_j - m_i|^2 in FP32 are each within their band of the FP64 values (the second up to
// 3.3 reMax, beyond which the test is off), so a difference above the sum of both bands
// (sideBand) decides.
struct SideF {
    float4 m;
    bool check;
};
__device__ __forceinline__ float4 posfOf(dvec4 p, const MpsParams& P) {
    return make_float4(d2fRN(p.x - P.domainMin[0]), d2fRN(p.y - P.domainMin[1]), d2fRN(p.z - P.domainMin[2]), 0.f);
}
__device__ __forceinline__ SideF sideF(const Dev& d, int i, dvec4 pi) {
    const SideCtx sc = sideCtx(d, i, pi);
    SideF s;
    s.check = sc.check;
    s.m = make_float4(0.f, 0.f, 0.f, 0.f);
    if (sc.check) s.m = posfOf(sc.mi, d.P);
    return s;
}
__device__ __forceinline__ bool sideOKF(const Dev& d, const SideF& s, float4 hj, float d2f, int i, int j) {
    if (!s.check) return true;
    const float t = dist2f(hj, s.m) - d2f;
    if (t > d.sideBand) return true;
    if (t < -d.sideBand) return false;
    return pairSideExact(d.pos, d.mirror, j, i);
}
// |x_j - x_i|^2 < R2 from the FP32 squared distance: certain outside [lo, hi]
__device__ __forceinline__ bool insideF(const Dev& d, float d2f, float lo, float hi, double R2, int i, int j) {
    if (d2f < lo) return true;
    if (d2f > hi) return false;
    return pairInsideExact(d.pos, j, i, R2);
}

// A pair vector and its squared norm for the sums (decisions are made before): the products
// are fused, one rounding less per term than the decision's expression.
__device__ __forceinline__ PairG pairSum(dvec4 pj, dvec4 pi) {
    PairG q;
    q.v0 = pj.x - pi.x; q.v1 = pj.y - pi.y; q.v2 = pj.z - pi.z;
    q.d2 = fma(q.v2, q.v2, fma(q.v1, q.v1, q.v0 * q.v0));
    return q;
}

// Bits of the entries k = l, l + L, ... < c of a list row that pass test(j, posf[j]); four
// entries' indices and FP32 copies are loaded ahead of their tests.
template <int L, class T>
__device__ __forceinline__ Mask rowMask(const Dev& d, const int* row, int l, int c, T&& test) {
    Mask m = maskNone();
    for (int k = l; k < c; k += 4 * L) {
        int jj[4];
        float4 hh[4];
#pragma unroll
        for (int u = 0; u < 4; u++) jj[u] = k + u * L < c ? ldStream(row + (size_t)(k + u * L) * d.N0) : -1;
#pragma unroll
        for (int u = 0; u < 4; u++) hh[u] = jj[u] >= 0 ? __ldg(&d.posf[jj[u]]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (jj[u] >= 0 && test(jj[u], hh[u])) maskSet(m, k + u * L);
    }
    return m;
}
// f(j, k) for the set bits of m in ascending order, the next entry's index loaded ahead.
template <class F>
__device__ __forceinline__ void forBits(const int* row, size_t N0, Mask m, F&& f) {
    int k = maskPop(m);
    if (k < 0) return;
    int j = ldStream(row + (size_t)k * N0);
    for (;;) {
        const int kn = maskPop(m);
        int jn = 0;
        if (kn >= 0) jn = ldStream(row + (size_t)kn * N0);
        f(j, k);
        if (kn < 0) break;
        k = kn; j = jn;
    }
}

// The per-entry weights of a list entry (element e) at squared distance d2: w(r; reS), w/r^2
// and, when the radii differ, w(r; reL).
__device__ __forceinline__ void storeWeights(const Dev& d, size_t e, double d2) {
    const MpsParams& P = d.P;
    double w, wd;
    weightR(d2, P.reS, P.weightType, w, wd);
    d.cw[e] = w;
    d.cwd[e] = wd;
    if (d.cwL) { double wl, wdl; weightR(d2, P.reL, P.weightType, wl, wdl); d.cwL[e] = wl; }
}

// The same for float-float sums, whose time is the latency of the gathers: ld(j) gathers what an
// entry needs and f(j, k, it) sums it; two entries' gathers are issued before their sums.  (The
// pressure gradient at 864k particles: 340 us entry by entry, 288 in twos, 354 to 376 with the
// next entry's gather held over a sum, which costs registers and so warps.)
template <class Ld, class F>
__device__ __forceinline__ void forBitsTwo(const int* row, size_t N0, Mask m, Ld&& ld, F&& f) {
    unsigned long long w = m.lo;
    for (int h = 0; h < 128; h += 64, w = m.hi)
        while (w) {
            const int k = __ffsll((long long)w) - 1 + h;
            w &= w - 1ull;
            const int j = ldStream(row + (size_t)k * N0);
            if (w) {
                const int k2 = __ffsll((long long)w) - 1 + h;
                w &= w - 1ull;
                const int j2 = ldStream(row + (size_t)k2 * N0);
                const auto a = ld(j), b = ld(j2);
                f(j, k, a);
                f(j2, k2, b);
            } else {
                f(j, k, ld(j));
            }
        }
}
// Entry by entry, for sums whose registers leave no room for a second entry.
template <class Ld, class F>
__device__ __forceinline__ void forBitsOne(const int* row, size_t N0, Mask m, Ld&& ld, F&& f) {
    unsigned long long w = m.lo;
    for (int h = 0; h < 128; h += 64, w = m.hi)
        while (w) {
            const int k = __ffsll((long long)w) - 1 + h;
            w &= w - 1ull;
            const int j = ldStream(row + (size_t)k * N0);
            f(j, k, ld(j));
        }
}

// f(j, e) for lane l's entries of a mask of row i, e the entry's ELL index.
template <int L, class F>
__device__ __forceinline__ void forMaskLane(const Dev& d, int i, Mask m, int l, F&& f) {
    forBits(d.nbr + i, d.N0, laneShare<L>(m, l), [&](int j, int k) { f(j, (size_t)k * d.N0 + i, k); });
}
// f(j, k) for the set bits of m by L lanes, bit t (counting set bits) going to lane t mod L:
// a mask of a few bits is shared evenly wherever they lie.
template <int L, class F>
__device__ __forceinline__ void forBitsShared(const int* row, size_t N0, Mask m, int l, F&& f) {
    for (int t = 0;; t++) {
        const int k = maskPop(m);
        if (k < 0) break;
        if ((t & (L - 1)) == l) f(ldStream(row + (size_t)k * N0), k);
    }
}

// The sweeps over the fluid particles near the polygon wall: a block takes 32 of the compacted
// list at a time, WALL_L lanes each.  The sums over a particle's mirror entries (up to a dozen)
// run on its lanes; what is done once per particle (the reflection about the wall plane, with
// its FP64 divisions and square root) runs on the first warp, one particle per lane, so its
// FP64 operations are issued once for 32 particles.  The wall pressure gradient took 415 us at
// 864k particles and 116 at 6.9k as one thread per particle testing its whole list: now 145
// and 30 (float-float 110 -> 90 us at 864k).
#define WALL_L 4
#define WALL_BLK 128
static inline int wallGrid(int n) { const int b = (n + 31) / 32; return b < 2432 ? b : 2432; }
// d.type/d.mask arrays of the near-wall list are those of the last k_side_masks.
template <class Pre, class Sum, class Post>
__device__ __forceinline__ void forNearWall(const Dev& d, Pre&& pre, Sum&& sum, Post&& post) {
    const int nn = *d.nearCount;
    for (int base = blockIdx.x * 32; base < nn; base += gridDim.x * 32) {
        const int own = base + (int)threadIdx.x;   // the first warp's particle
        const bool head = threadIdx.x < 32 && own < nn;
        if (head) pre(d.nearList[own], (int)threadIdx.x);
        __syncthreads();
        const int g = threadIdx.x / WALL_L, l = threadIdx.x & (WALL_L - 1);
        if (base + g < nn) sum(d.nearList[base + g], g, l);
        __syncthreads();
        if (head) post(d.nearList[own], (int)threadIdx.x);
        __syncthreads();
    }
}

// Mirror entries of the near-wall particles at positions that have no list (the shifting's wall
// term, whose first sweep has just moved them).  A warp takes 8 of the block's 32 particles one
// after another and tests a particle's candidates with all its lanes: the start-of-step skin
// list while that covers the particle (skin: the flag of the last k_skin_check), else the nine
// bucket rows of its window.  The entries are left in cand[g] in scan order, their number in
// num[g] (-1: more than WALL_CAND); the caller synchronises, then forWallCand walks them.
#define WALL_CAND 128
struct WallCand {
    int cand[32][WALL_CAND];
    int num[32];
};
__device__ __forceinline__ void wallCandidates(const Dev& d, WallCand& W, int base, int nn, bool skin) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const MpsParams& P = d.P;
    for (int q = 0; q < 8; q++) {
        const int g = warp * 8 + q;
        if (base + g >= nn) break;
        const int i = d.nearList[base + g];
        const dvec4 pi = d.pos[i];
        const float4 fi = d.posf[i], mf = posfOf(d.mirror[i], P);
        int cnt = 0;
        auto test = [&](int j, float4 fj) {
            const float d2f = dist2f(fj, fi);
            if (d2f > d.bandHiS || j == i) return false;
            const float dm2f = dist2f(fj, mf);
            if (dm2f > d.bandHiS) return false;
            if (!insideF(d, d2f, d.bandLoS, d.bandHiS, P.reS2, i, j)) return false;
            if (!(dm2f < d.bandLoS) && !mirrorInsideExact(d.pos, d.mirror, j, i, P.reS2)) return false;
            const float t = dm2f - d2f;
            if (t > d.sideBand) return true;
            if (t < -d.sideBand) return false;
            return pairSideExact(d.pos, d.mirror, j, i);
        };
        auto append = [&](bool in, int j) {
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int k = cnt + __popc(m & ((1u << lane) - 1u));
            if (in && k < WALL_CAND) W.cand[g][k] = j;
            cnt += __popc(m);
        };
        const int c = skin ? d.skinCnt[i] : d.K + 1;
        if (c <= d.K && d.skinCell[i] == cellKeyOf(d, pi, fi)) {
            for (int k0 = 0; k0 < c; k0 += 32) {
                bool in = false;
                int j = i;
                if (k0 + lane < c) {
                    j = ldStream(d.skinNbr + (size_t)(k0 + lane) * d.N0 + i);
                    in = test(j, __ldg(&d.posf[j]));
                }
                append(in, j);
            }
        } else {
            int ix, iy, iz;
            bucketCoordsHi(d, pi, fi, ix, iy, iz);
            const int nr = d.dz3 ? 9 : 3;
            int a = 0, b = 0;
            if (lane < nr) {
                const long long jb = (long long)((iz - 1) * d.dz3 + lane / 3) * P.numBucketsXY +
                                     (long long)(iy - 1 + lane % 3) * P.numBucketsX + ix;
                const long long lo = jb - 1 > 0 ? jb - 1 : 0, hi = jb + 1 < d.nB - 1 ? jb + 1 : d.nB - 1;
                if (lo <= hi) { a = d.cellStart[lo]; b = d.cellStart[hi + 1]; }
            }
            for (int r = 0; r < nr; r++) {
                const int s0 = __shfl_sync(0xffffffffu, a, r), s1 = __shfl_sync(0xffffffffu, b, r);
                for (int t = s0; t < s1; t += 32) {
                    bool in = false;
                    int j = i;
                    if (t + lane < s1) {
                        j = __ldg(d.cellSorted + t + lane);
                        in = test(j, __ldg(&d.posf[j]));
                    }
                    append(in, j);
                }
            }
        }
        if (lane == 0) W.num[g] = cnt <= WALL_CAND ? cnt : -1;
    }
}
// f(j) for lane l's share of the mirror entries of particle i = the block's g-th; one lane scans
// the buckets for a particle with more entries than were kept.
template <class F>
__device__ __forceinline__ void forWallCand(const Dev& d, const WallCand& W, int i, int g, int l, F&& f) {
    const int n = W.num[g];
    for (int t = l; t < n; t += WALL_L) f(W.cand[g][t]);
    if (n >= 0 || l != 0) return;
    const dvec4 pi = d.pos[i], mi = d.mirror[i];
    forCells(d, pi, [&](int j) {
        const dvec4 pj = d.pos[j];
        const double d2 = pairOf(pj, pi).d2, dm2 = pairMirror(pj, mi).dm2;
        if (j != i && d2 < d.P.reS2 && dm2 < d.P.reS2 && d2 < dm2) f(j);
    });
}

// End of the shifting's wall term at particle i (src/MpsShifting.cpp:640-691): its own image,
// the reflection, and the shift of inner particles.
__device__ __forceinline__ void wallGradConcEnd(const Dev& d, int i, double dx, double dy, double dz) {
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i], mi = d.mirror[i];
    const ReflG r = makeRefl(pi, mi, P.epsilonZero, true);
    const double ci = d.conc[i];
    const PairM s = pairMirror(pi, mi);
    if (s.dm2 < P.reS2) {
        const double f = (ci + ci) * wfun(sqrt(s.dm2), P.reS, P.weightType) / s.dm2;
        dx += f * s.m0; dy += f * s.m1; dz += f * s.m2;
    }
    const double g0 = -(r.R[0] * dx + r.R[1] * dy + r.R[2] * dz) * P.coeffPressGrad;
    const double g1 = -(r.R[3] * dx + r.R[4] * dy + r.R[5] * dz) * P.coeffPressGrad;
    const double g2 = -(r.R[6] * dx + r.R[7] * dy + r.R[8] * dz) * P.coeffPressGrad;
    dvec4 g = d.gradC[i];
    g.x += g0; g.y += g1; g.z += g2;
    d.gradC[i] = g;
    d.shift[i] = d.bc[i] == P.inner
                     ? make_dvec4(-P.coeffShifting2 * g0, -P.coeffShifting2 * g1, -P.coeffShifting2 * g2, 0.0)
                     : make_dvec4(0, 0, 0, 0);
}
