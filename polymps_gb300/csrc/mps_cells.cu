// mps_cells.cu — bucket list (MpsBucket::updateParticlesID, src/MpsBucket.cpp:299-353) as
// a counting sort, and the ELL neighbour list of the current positions through that
// stale list (the 27-bucket scan shared by every operator, e.g. src/MpsPndNeigh.cpp:209-258).
//
// Both are HBM/L2-latency bound integer work: one coalesced pass over the particles for
// the bucket keys, atomics into the per-bucket counters, a device-wide scan, a scatter
// and a ranking within each bucket that restores ascending particle order (the
// reference's linked lists are filled in ascending index order).
#include <atomic>
#include "mps_df.cuh"
#include "mps_internal.h"
#include "mps_lanes.cuh"

static std::atomic<long long> g_launches{0};
void countLaunch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launchCount() { return g_launches.load(std::memory_order_relaxed); }

// ------------------------------------------------------------------ bucket keys
// Warp-level counting: the lanes of a warp that share a bucket key (most of them, since the
// storage is kept in bucket order) form one group; its lowest lane adds the group's size to
// the bucket's counter (or cursor) and every lane's place is the group's base plus its rank
// among the group's lanes (lane order = particle order).  Returns that place.
__device__ __forceinline__ int warpGroupAdd(int* counters, int key, bool active) {
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!active) return -1;
    const unsigned grp = __match_any_sync(act, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(grp) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counters + key, __popc(grp));
    base = __shfl_sync(grp, base, leader);
    return base + __popc(grp & ((1u << lane) - 1u));
}

// One bucket coordinate of updateParticlesID: (int)((x - min) * inv) in 3D,
// (int)((x - min) * inv + eps) in 2D, with dx = x - min (exact FP64 subtraction, the
// reference's first operation).  The FP32 product of the particle's FP32 copy h = fl32(dx)
// and fl32(inv) lies within 3 * 2^-24 relative of the FP64 one, so its truncation is exact
// unless it is within a margin of an integer (or below it); those rare cases evaluate the
// FP64 expression out of line (inlined, the compiler would predicate it into every thread).
static __device__ __noinline__ int bucketKeyCoordExact(double dx, double inv, double eps, bool withEps) {
    const double q = xmul(dx, inv);
    return (int)(withEps ? xadd(q, eps) : q);
}
__device__ __forceinline__ int bucketKeyCoord(float h, double dx, float invf, float epsf, double inv, double eps,
                                              bool withEps) {
    const float q = withEps ? fmaf(h, invf, epsf) : h * invf;
    const float m = 5e-7f * fabsf(q) + 1e-6f;
    const float f = q - floorf(q);
    if (q > m && f > m && f < 1.0f - m) return (int)q;
    return bucketKeyCoordExact(dx, inv, eps, withEps);
}

// 2D adds epsilonZero, 3D does not (src/MpsBucket.cpp:312-313 vs :333-335); ghosts skipped.
// Every lane of a warp reaches the warp-level count (lanes past N0 take part without a key).
__global__ void k_cell_key(Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = liveN(d);
    int key = -1;
    if (i < n && d.type[i] == d.P.ghost) {
        key = d.nB;   // live, in no bucket: listed after the buckets, never scanned
    } else if (i < n) {
        const MpsParams& P = d.P;
        dvec4 p = d.pos[i];
        // x - min once: the key's first operation and the FP32 copies' argument
        const double dx = xsub(p.x, P.domainMin[0]), dy = xsub(p.y, P.domainMin[1]), dzz = xsub(p.z, P.domainMin[2]);
        const df fx = dfD(dx), fy = dfD(dy), fz = dfD(dzz);
        const float4 hi = make_float4(fx.h, fy.h, fz.h, 0.f);
        const bool two = (int)P.dim == 2;
        int ix = bucketKeyCoord(hi.x, dx, d.invSidef, d.epsf, P.invBucketSide, P.epsilonZero, two);
        int iy = bucketKeyCoord(hi.y, dy, d.invSidef, d.epsf, P.invBucketSide, P.epsilonZero, two);
        int iz = two ? 0 : bucketKeyCoord(hi.z, dzz, d.invSidef, d.epsf, P.invBucketSide, P.epsilonZero, false);
        long long ib = (long long)iz * P.numBucketsXY + (long long)iy * P.numBucketsX + ix;
        if (ib < 0 || ib >= d.nB) {
            setErr(d, MPSE_DOMAIN);
            key = d.nB;
        } else {
            key = (int)ib;
        }
        // FP32 copy of the start-of-step positions for the prefiltered scans (hi, lo parts)
        d.posf[i] = hi;
        d.posLo[i] = make_float4(fx.l, fy.l, fz.l, 0.f);
    }
    warpGroupAdd(d.cellCount, key, key >= 0);
    if (i < d.N0) d.cellOf[i] = key;
}

// The records (reference index, slot) of each bucket in arrival order.
__global__ void k_cell_scatter(Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = (i < d.N0) ? d.cellOf[i] : -1;
    const int r = warpGroupAdd(d.cellCursor, c, c >= 0);
    if (c >= 0) d.cellRec[d.cellStart[c] + r] = make_int2(d.orig[i], i);
    else if (i < d.N0) d.cellPos[i] = -1;
}

// Each bucket ordered by reference index (the reference's linked-list order; buckets hold ~10
// particles), the range after the last bucket the same way: a record's place is the number of
// smaller reference indices in its bucket, so every particle finds its own with a few reads
// of neighbouring records: 6 us at 6.9k particles and 15 at 864k, with the inverse list and the
// copies below (one thread sorting each bucket by insertion walked dependent loads: 28 and 52
// us, and two more launches).  place: also the inverse list and the FP32 copies in
// bucket order (the renumbering, which moves the slots, writes them after it).
// The counters and cursors are cleared for the next build.
__global__ void k_cell_rank(Dev d, bool place) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = p; k < 2 * (d.nB + 2); k += gridDim.x * blockDim.x) d.cellCount[k] = 0;
    if (p >= d.cellStart[d.nB + 1]) return;
    const int2 me = d.cellRec[p];
    const int c = d.cellOf[me.y];
    const int s0 = d.cellStart[c], s1 = d.cellStart[c + 1];
    int at = s0;
    for (int q = s0; q < s1; q++) at += d.cellRec[q].x < me.x ? 1 : 0;
    d.cellSorted[at] = me.y;
    if (!place) return;
    d.cellPos[me.y] = at;
    if (c < d.nB) {
        d.posfCell[at] = d.posf[me.y];
        d.posLoCell[at] = d.posLo[me.y];
    }
}

// ------------------------------------------------------------------ exclusive scan
// Block scan for int arrays: tiles, then each tile's offset from the tile sums before it.
#define SCAN_BLOCK 1024
#define SCAN_PER_THREAD 4
#define SCAN_TILE (SCAN_BLOCK * SCAN_PER_THREAD)

__device__ __forceinline__ int blockExclusiveScan(int v, int* smem, int& total) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < (int)(blockDim.x >> 5)) ? smem[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        smem[lane] = w;
    }
    __syncthreads();
    int warpPrefix = (warp > 0) ? smem[warp - 1] : 0;
    total = smem[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warpPrefix + x - v;
}

__global__ void k_scan_tiles(const int* in, int* out, int* tileSums, int n) {
    __shared__ int smem[32];
    int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
    int v[SCAN_PER_THREAD];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; k++) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        s += v[k];
    }
    int total;
    int pre = blockExclusiveScan(s, smem, total);
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; k++) {
        if (base + k < n) out[base + k] = pre;
        pre += v[k];
    }
    if (threadIdx.x == 0 && tileSums) tileSums[blockIdx.x] = total;
}

// out += the sums of the tiles before this block's; the last block writes the total to out[n].
__global__ void k_scan_add(int* out, const int* tileSums, int n) {
    __shared__ int smem[32];
    int add = 0;
    for (int t = threadIdx.x; t < (int)blockIdx.x; t += SCAN_BLOCK) add += tileSums[t];
    int total;
    blockExclusiveScan(add, smem, total);
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; k++)
        if (base + k < n) out[base + k] += total;
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = total + tileSums[blockIdx.x];
}
// Up to SCAN_SMALL tiles by one block, a tile after the other (one launch for three).
#define SCAN_SMALL 4
__global__ void k_scan_small(const int* in, int* out, int n) {
    __shared__ int smem[32];
    int carry = 0;
    for (int t = 0; t < n; t += SCAN_TILE) {
        const int base = t + threadIdx.x * SCAN_PER_THREAD;
        int v[SCAN_PER_THREAD], s = 0, total;
#pragma unroll
        for (int k = 0; k < SCAN_PER_THREAD; k++) { v[k] = (base + k < n) ? in[base + k] : 0; s += v[k]; }
        int pre = carry + blockExclusiveScan(s, smem, total);
#pragma unroll
        for (int k = 0; k < SCAN_PER_THREAD; k++) {
            if (base + k < n) out[base + k] = pre;
            pre += v[k];
        }
        carry += total;
    }
    if (threadIdx.x == 0) out[n] = carry;
}

// out[0..n) = exclusive scan of in; out[n] = total.  scratch holds >= tiles ints.
void scanExclusive(const int* in, int* out, int n, int* scratch, cudaStream_t s) {
    int tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (tiles <= SCAN_SMALL) {
        k_scan_small<<<1, SCAN_BLOCK, 0, s>>>(in, out, n);
        return;
    }
    k_scan_tiles<<<tiles, SCAN_BLOCK, 0, s>>>(in, out, scratch, n);
    k_scan_add<<<tiles, SCAN_BLOCK, 0, s>>>(out, scratch, n);
}
int scanScratchInts(int n) { return 2 * ((n + SCAN_TILE - 1) / SCAN_TILE) + 4; }

// ------------------------------------------------------------------ renumbering
// Storage renumbering into the order of the bucket list just built: slot s receives the
// particle listed at s (live particles; slots beyond the live count keep theirs), every
// per-particle array is gathered through a scratch buffer, the reference-index maps follow,
// and the list becomes the identity.  Neighbours are then stored next to each other, which
// is what the gathers of every sweep and the coalescing of the bucket-order scans want.
// Two launches: all arrays gathered into the weight cache of the list (K doubles per particle,
// twice; the bucket rebuild has just made the list stale), then copied back, with the maps, the
// inverse list and the bucket-ordered copies of the new order.  (A launch and a copy per array were
// 84 launches of 2 to 30 us.)
#define PERM_V 16
#define PERM_S 18
#define PERM_I 6
struct PermArrays {
    dvec4* v[PERM_V];
    double* s[PERM_S];
    int* i[PERM_I];
};
static PermArrays permArrays(const Dev& d) {
    return {{d.pos, d.vel, d.acc, d.accStar, d.mirror, d.wallPos, d.polyNormal, d.normal, d.npcd, d.gradC, d.forceWall, d.c1,
             d.c2, d.c3, d.dvel, d.shift},
            {d.press, d.pressPPE, d.pressPPEprev, d.pressPPEprev2, d.pndi, d.pndki, d.pndski, d.pndSmall, d.npcd2, d.conc,
             d.velDiv, d.diffTerm, d.pndWall, d.riw2, d.devDot, d.source, d.aux1, d.aux2},
            {d.type, d.bc, d.numNeigh, d.nNeighWall, d.nearWall, d.cellOf}};
}
// scratch: vectors in cw, the rest in cwd (each K doubles a particle)
static_assert(PERM_V * sizeof(dvec4) <= NBR_CAP_2D * sizeof(double) && NBR_CAP_2D <= NBR_CAP_3D, "cw holds the vectors");
static_assert(2 * sizeof(float4) + PERM_S * sizeof(double) + (PERM_I + 1) * sizeof(int) <= NBR_CAP_2D * sizeof(double),
              "cwd holds the FP32 copies, the scalars, the integers and the reference index");
struct PermScratch {
    dvec4* v;
    float4 *hi, *lo;
    double* s;
    int* i;
};
__host__ __device__ __forceinline__ PermScratch permScratch(const Dev& d) {
    const size_t n = d.N0;
    PermScratch t;
    t.v = reinterpret_cast<dvec4*>(d.cw);
    t.hi = reinterpret_cast<float4*>(d.cwd);
    t.lo = t.hi + n;
    t.s = reinterpret_cast<double*>(t.lo + n);
    t.i = reinterpret_cast<int*>(t.s + PERM_S * n);
    return t;
}
__global__ void k_perm_gather(Dev d, PermArrays a) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.N0) return;
    const size_t n = d.N0;
    const int p = (s < *d.nLive) ? d.cellSorted[s] : s;
    const PermScratch t = permScratch(d);
#pragma unroll
    for (int k = 0; k < PERM_V; k++) t.v[k * n + s] = a.v[k][p];
    t.hi[s] = d.posf[p];
    t.lo[s] = d.posLo[p];
#pragma unroll
    for (int k = 0; k < PERM_S; k++) t.s[k * n + s] = a.s[k][p];
#pragma unroll
    for (int k = 0; k < PERM_I; k++) t.i[k * n + s] = a.i[k][p];
    t.i[PERM_I * n + s] = d.orig[p];
}
__global__ void k_perm_place(Dev d, PermArrays a) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.N0) return;
    const size_t n = d.N0;
    const PermScratch t = permScratch(d);
#pragma unroll
    for (int k = 0; k < PERM_V; k++) a.v[k][s] = t.v[k * n + s];
    const float4 hi = t.hi[s], lo = t.lo[s];
    d.posf[s] = hi;
    d.posLo[s] = lo;
#pragma unroll
    for (int k = 0; k < PERM_S; k++) a.s[k][s] = t.s[k * n + s];
#pragma unroll
    for (int k = 0; k < PERM_I; k++) a.i[k][s] = t.i[k * n + s];
    const int r = t.i[PERM_I * n + s];
    d.orig[s] = r;
    d.slotOf[r] = s;
    if (s < *d.nLive) d.cellSorted[s] = s;
    d.cellPos[s] = s < d.cellStart[d.nB + 1] ? s : -1;
    if (s < d.cellStart[d.nB]) {
        d.posfCell[s] = hi;
        d.posLoCell[s] = lo;
    }
}
int renumberLaunches() { return 2; }
static void launchRenumber(const Dev& d, cudaStream_t s) {
    const PermArrays a = permArrays(d);
    k_perm_gather<<<gridFor(d.N0, 256), 256, 0, s>>>(d, a);
    k_perm_place<<<gridFor(d.N0, 256), 256, 0, s>>>(d, a);
}

void launchBuckets(const Dev& d, int* scanScratch, cudaStream_t s, bool renumber) {
    k_cell_key<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    scanExclusive(d.cellCount, d.cellStart, d.nB + 1, scanScratch, s);
    k_cell_scatter<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    k_cell_rank<<<gridFor(d.N0, 256), 256, 0, s>>>(d, !renumber);
    if (renumber) launchRenumber(d, s);
}

// ------------------------------------------------------------------ FP32 copy
__global__ void k_posf(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N0) return;   // every slot: stale bucket entries may name removed particles
    float4 hi, lo;
    splitPos(d.pos[i], d.P, hi, lo);
    d.posf[i] = hi;
    d.posLo[i] = lo;
}

// The copies and, for the list filter that follows, the skin list's validity (k_skin_check) and
// the filter's cleared counters, in one pass.
__global__ void k_posf_check(Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) { *d.rescan = 0; d.counters[0] = 0ull; }
    if (i >= d.N0) return;
    float4 hi, lo;
    splitPos(d.pos[i], d.P, hi, lo);
    d.posf[i] = hi;
    d.posLo[i] = lo;
    if (i < liveN(d) && !(dist2f(hi, d.posSkin[i]) <= d.skinMove2)) d.skinFlag[0] = 1;
}
void launchPosfCheck(const Dev& d, cudaStream_t s) { k_posf_check<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }

// ------------------------------------------------------------------ neighbour list
// FP32 copy of the positions in bucket order, refreshed whenever positions change.
__global__ void k_posf_cell(Dev d) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.cellStart[d.nB]) return;
    int j = d.cellSorted[s];
    d.posfCell[s] = d.posf[j];
    d.posLoCell[s] = d.posLo[j];
}
void launchPosfCell(const Dev& d, cudaStream_t s) {
    k_posf_cell<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
}
void launchPosfOnly(const Dev& d, cudaStream_t s) { k_posf<<<gridFor(d.N0, 256), 256, 0, s>>>(d); }
void launchPosf(const Dev& d, cudaStream_t s) {
    k_posf<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
    launchPosfCell(d, s);
}

// The 27-bucket scan into list rows, L lanes per particle: the three buckets of a row of the
// window are one range of the bucket order (about 28 particles), tested 32 candidates at a time
// into a bit mask whose set bits are then appended in scan order (appended where they are
// found, every warp issued the append for nearly every candidate).  The skin list: 74 -> 19 us
// at 6.9k particles (8 lanes), 98 -> 71 at 108k, 1,675 -> 1,311 at 2.8M (366 and 394 at 864k).
//   MODE 0: the start-of-step skin list: candidates within reMax + skin (FP32 test against a
//     radius that includes the rounding band: a superset of every list the step's sweeps can
//     need while the particles stay within half the skin), start position and scan window.
//   MODE 1: the list of the current positions.  Candidates are decided in FP32 first; only
//     those whose FP32 squared distance falls in the rounding band around the list radius^2 are
//     re-tested in exact FP64, so membership equals the reference's test dst^2 < re^2.
//   MODE 2: the same with the entries' weights for the epoch, in a second pass over the members
//     (formed where a candidate is accepted, they took 721 us for 158 at 108k particles): the
//     FP64 divisions and square roots of all later sweeps happen here once.
template <int MODE, int L>
__global__ void __launch_bounds__(128) k_build_list(Dev d) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const dvec4 pi = d.pos[i];
    const float4 fi = d.posf[i];
    const size_t N0 = d.N0;
    const int me = d.cellPos[i];   // the particle is no neighbour of itself
    int cnt = 0;
    int ix, iy, iz;
    bucketCoordsHi(d, pi, fi, ix, iy, iz);
    const int minZ = (iz - 1) * d.dz3, maxZ = (iz + 1) * d.dz3;
#pragma unroll 1
    for (int jz = minZ; jz <= maxZ; jz++)
#pragma unroll 1
        for (int jy = iy - 1; jy <= iy + 1; jy++) {
            const long long jb = (long long)jz * P.numBucketsXY + (long long)jy * P.numBucketsX + ix;
            const long long lo = jb - 1 > 0 ? jb - 1 : 0, hi = jb + 1 < d.nB - 1 ? jb + 1 : d.nB - 1;
            if (lo > hi) continue;
            const int s1 = d.cellStart[hi + 1];
#pragma unroll 1
            for (int s0 = d.cellStart[lo]; s0 < s1; s0 += 32) {
                // bit b: candidate s0 + b.  Every lane's bit positions are constants and nothing is
                // predicated: what lies past the range (the array is padded) is masked off
                // after, like the particle itself, so a candidate costs nine instructions
                const int w = s1 - s0;
                const float4* const f = d.posfCell + s0 + l;
                unsigned m = 0u, sure = 0u;
#pragma unroll
                for (int g = 0; g < 32 / L; g += 4) {
                    if (g * L >= w) break;
                    float4 h[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) h[u] = __ldg(f + (g + u) * L);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float d2f = dist2f(h[u], fi);
                        if (!(d2f > (MODE == 0 ? d.skinR2 : d.bandHi))) m |= 1u << ((g + u) * L);
                        if (MODE != 0 && d2f < d.bandLo) sure |= 1u << ((g + u) * L);
                    }
                }
                if (L > 1) { m <<= l; sure <<= l; }
                if (w < 32) m &= (1u << w) - 1u;
                if ((unsigned)(me - s0) < 32u) m &= ~(1u << (me - s0));
                if (MODE != 0)
                    for (unsigned r = m & ~sure; r; r &= r - 1u) {   // inside the band: FP64 decides
                        const int b = __ffs((int)r) - 1;
                        if (!pairInsideExact(d.pos, __ldg(d.cellSorted + s0 + b), i, d.reMax2)) m &= ~(1u << b);
                    }
                if (L == 1) {
                    for (; m; m &= m - 1u, cnt++)
                        if (cnt < d.K) d.nbr[(size_t)cnt * N0 + i] = __ldg(d.cellSorted + s0 + __ffs((int)m) - 1);
                } else {
                    unsigned all = m;
#pragma unroll
                    for (int o = 1; o < L; o <<= 1) all |= __shfl_xor_sync(laneGroup<L>(), all, o);
                    for (; m; m &= m - 1u) {
                        const int b = __ffs((int)m) - 1;
                        const int k = cnt + __popc(all & ((1u << b) - 1u));
                        if (k < d.K) d.nbr[(size_t)k * N0 + i] = __ldg(d.cellSorted + s0 + b);
                    }
                    cnt += __popc(all);
                }
            }
        }
    if (MODE == 0) {
        if (i == 0 && l == 0) d.skinFlag[0] = 0;
        if (l == 0) {
            d.nbrCount[i] = cnt > d.K ? d.K + 1 : cnt;   // K + 1: the row overflowed, rescanned where read
            d.posSkin[i] = fi;
            d.skinCell[i] = cellKeyOf(d, pi, fi);
        }
        return;
    }
    const int c = cnt < d.K ? cnt : d.K;
    if (l == 0) {
        if (cnt > d.K) setErr(d, MPSE_CAPACITY);
        d.nbrCount[i] = c;
    }
    warpCount(d.counters, l == 0 ? (unsigned)c : 0u);
    if (MODE == 2) {
        __syncwarp(laneGroup<L>());
        for (int k = l; k < c; k += L) {
            const size_t e = (size_t)k * N0 + i;
            storeWeights(d, e, pairSum(d.pos[d.nbr[e]], pi).d2);
        }
    }
}
template <int MODE>
static void launchBuild(const Dev& d, cudaStream_t s) {
#define LAUNCH(L) k_build_list<MODE, L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// Per-entry weights of the current list for the FP64 sweeps, when the list was built by
// the DF32 tier (which stores none); the same expressions as k_build_list.
__global__ void __launch_bounds__(128) k_fill_cache(Dev d) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    dvec4 pi = d.pos[i];
    int c = d.nbrCount[i];
    for (int k = 0; k < c; k++) {
        size_t e = (size_t)k * d.N0 + i;
        storeWeights(d, e, pairSum(d.pos[d.nbr[e]], pi).d2);
    }
}
void launchFillCache(const Dev& d, cudaStream_t s) {
    k_fill_cache<<<gridFor(d.N0, 128), 128, 0, s>>>(d);
}

void launchNeighborList(const Dev& d, cudaStream_t s, bool weights) {
    cudaMemsetAsync(d.counters, 0, sizeof(unsigned long long), s);
    launchPosf(d, s);
    if (weights) launchBuild<2>(d, s);
    else launchBuild<1>(d, s);
}
void launchSkinList(const Dev& d, cudaStream_t s) {
    launchBuild<0>(d, s);
}

// ------------------------------------------------------------------ entry masks
// After the wall pass: for each particle, which entries are inside the reS / reL ball and
// not on the mirror side (dstij2 < dstimj2, e.g. src/MpsPndNeigh.cpp:249), with the
// reference's decisions: from the FP32 copies outside their rounding bands, in FP64 inside
// them.  Particles whose mirror is far (see SideCtx) and whose list radius equals the ball
// radius take every entry without per-entry work.  Fluid particles near the wall also get
// their mirror entries and are appended to nearList for the wall-only sweeps, which walk the
// masks instead of testing the list again.
template <int L>
__global__ void __launch_bounds__(128) k_side_masks(Dev d, int* oldCount) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i == 0 && l == 0) *oldCount = 0;   // the next call's counter
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    const int c = d.nbrCount[i];
    const Mask all = maskFirst(c);
    const dvec4 pi = d.pos[i];
    const bool near = P.wallType == 1 && d.type[i] == P.fluid && d.nearWall[i];
    SideF sd = sideF(d, i, pi);
    if (near && !sd.check) sd.m = posfOf(d.mirror[i], P);
    const bool fullS = P.reS2 >= d.reMax2, fullL = P.reL2 >= d.reMax2;
    const bool two = d.mirrorL != d.mirrorS;
    Mask mS = all, mL = all;
    if (sd.check || near || !fullS || !fullL) {
        mS = maskNone(); mL = maskNone();
        Mask rS = maskNone(), rL = maskNone();
        const float4 fi = d.posf[i];
        const int* row = d.nbr + i;
        auto mirrorIn = [&](float dm2f, float lo, float hi, double R2, int j) {
            if (dm2f < lo) return true;
            if (dm2f > hi) return false;
            return mirrorInsideExact(d.pos, d.mirror, j, i, R2);
        };
        for (int k = l; k < c; k += L) {
            const int j = ldStream(row + (size_t)k * d.N0);
            const float4 fj = __ldg(&d.posf[j]);
            const float d2f = dist2f(fj, fi);
            if (!sideOKF(d, sd, fj, d2f, i, j)) continue;
            const bool inS = fullS || insideF(d, d2f, d.bandLoS, d.bandHiS, P.reS2, i, j);
            const bool inL = fullL || insideF(d, d2f, d.bandLoL, d.bandHiL, P.reL2, i, j);
            if (inS) maskSet(mS, k);
            if (inL) maskSet(mL, k);
            if (near) {
                const float dm2f = dist2f(fj, sd.m);
                if (inS && mirrorIn(dm2f, d.bandLoS, d.bandHiS, P.reS2, j)) maskSet(rS, k);
                if (two && inL && mirrorIn(dm2f, d.bandLoL, d.bandHiL, P.reL2, j)) maskSet(rL, k);
            }
        }
        mS = laneOr<L>(mS); mL = laneOr<L>(mL);
        if (near) {
            rS = laneOr<L>(rS);
            if (two) rL = laneOr<L>(rL);
            if (l == 0) {
                d.mirrorS[i] = rS;
                if (two) d.mirrorL[i] = rL;
            }
        }
    }
    if (l == 0) {
        d.maskS[i] = mS;
        d.maskL[i] = mL;
        if (near) d.nearList[atomicAdd(d.nearCount, 1)] = i;
    }
}

void launchSideMasks(const Dev& d, int* oldCount, cudaStream_t s) {
#define LAUNCH(L) k_side_masks<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d, oldCount)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// nearList for the current positions, where no list and no masks are built
__global__ void k_near_list(Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < liveN(d) && d.type[i] == d.P.fluid && d.nearWall[i]) d.nearList[atomicAdd(d.nearCount, 1)] = i;
}
void launchNearList(const Dev& d, cudaStream_t s) {
    cudaMemsetAsync(d.nearCount, 0, sizeof(int), s);
    k_near_list<<<gridFor(d.N0, 256), 256, 0, s>>>(d);
}
