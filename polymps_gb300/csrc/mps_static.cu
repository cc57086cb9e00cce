// mps_static.cu — allocation-free Jacobi-preconditioned CG on a caller-supplied CSR system.
//
// Some callers cannot allocate device memory at the moment they need a pressure solve:
// a host application that runs inside a memory budget owned by another framework (its
// caching allocator must see every byte, and a raw cudaMalloc would bypass or fragment
// it), a real-time stepping loop that forbids allocation latency once running, or a plugin
// called back from a library that hands it only the arrays it owns.  For them this entry
// point keeps all of its working vectors in one file-scope device array reserved when the
// library is loaded: it calls no cudaMalloc/cudaFree and no allocating library routine.
//
// Limits and rules (the same as in the declaration in mpsgpu.h):
//  * at most MPSGPU_STATIC_MAX_ROWS rows; larger systems are rejected with an error;
//  * the array is shared by every call on a device and keeps the last call's contents:
//    each call clears the words it relies on, and calls of several host threads take turns
//    (a call returns when its work on the GPU is done);
//  * the first call on a device looks the array's device address up (with that device
//    current); make that first call before any stream capture begins.
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <cuda_runtime.h>
#include "../../include/mpsgpu.h"
#include "mps_grid.cuh"

#define SBLOCKS 256   // blocks at most (one per SM)
#define SBLK 512
#define SLANES 4      // lanes of a row in the matrix products
#define SROW 12       // entries of a lane in flight
#define SMAX MPSGPU_STATIC_MAX_ROWS

// layout in doubles: z (SMAX), r, p, Ap, inverse diagonal (SMAX each; only where the block's
// rows do not fit its shared memory), scalars (16), control words (8 unsigned ints), the grid
// barrier's arrivals (a 128-byte line of its own), the grid sums' partials (2 sets of GRID_NV values)
#define OFF_Z 0
#define OFF_VEC (1ull * SMAX)
#define OFF_SCAL (5ull * SMAX)
#define OFF_CTRL (OFF_SCAL + 16ull)
#define OFF_ARR (OFF_SCAL + 32ull)
#define OFF_PART (OFF_ARR + 16ull)
#define SCRATCH_DOUBLES (OFF_PART + 2ull * GRID_NV * SBLOCKS)

// The scratch every call uses (about 5.3 MB per GPU, held from library load until exit).
static __device__ __align__(256) double g_pcgScratch[SCRATCH_DOUBLES];

enum { SC_BB = 0, SC_RR0 };
// control words: [1] 1 converged or nothing to do, 2 stopped at the iteration cap,
// [2] iterations, [3] breakdown, [4] UINT_MAX - (lowest row without a usable diagonal) or 0,
// [5] a grid wait ran out
enum { C_DONE = 1, C_ITERS, C_BREAK, C_BADROW, C_ABORT };

namespace {

// NV sums over the grid, then fin(sums) on one thread of each block (the same bits in every
// block), whose writes to shared memory every thread of the block sees on return.  The
// FP64 pipe takes 2 lanes per clock and SM, 16 clocks per warp instruction: the block's tree
// halves the active warps in shared memory (20 warp additions of a 512-thread block, 16
// shuffle trees would take 80), and the scalars' divisions run on one warp, not on 32.
template <int NV, class Fin>
__device__ bool gridTotal(double (&v)[NV], GridBar& g, unsigned long long* part, int active, Fin&& fin) {
    __shared__ double sm[NV][SBLK];   // level w's values at [w, 2 w)
    const int t = threadIdx.x;
    g.gen++;
#pragma unroll
    for (int w = SBLK / 2; w >= 32; w >>= 1) {
        if (w >= active) continue;   // only the threads below `active` hold anything
        if (t >= w && t < 2 * w)
#pragma unroll
            for (int q = 0; q < NV; q++) sm[q][t] = v[q];
        __syncthreads();
        if (t < w)
#pragma unroll
            for (int q = 0; q < NV; q++) v[q] += sm[q][t + w];
    }
    __syncthreads();
    int ok = 1;
    if (t < 32) {
        unsigned long long pv[NV], got[NV][GRID_PER_LANE];
#pragma unroll
        for (int q = 0; q < NV; q++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
            pv[q] = (unsigned long long)__double_as_longlong(v[q]);
        }
        ok = gridCollectWarp0<NV>(pv, g, part, 0ull, got);
        if (ok) {
#pragma unroll
            for (int q = 0; q < NV; q++) {
                double a[GRID_PER_LANE];
#pragma unroll
                for (int m = 0; m < GRID_PER_LANE; m++) a[m] = __longlong_as_double((long long)got[q][m]);
                double s = a[0];
                if (gridDim.x > 32) s = (s + a[1]) + (a[2] + a[3]);
                if (gridDim.x > 128) s += (a[4] + a[5]) + (a[6] + a[7]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                v[q] = s;
            }
            if (t == 0) fin(v);
        }
    }
    return __syncthreads_and(ok) != 0;
}

// Row sums of SLANES consecutive rows (row0 ..) by the SLANES lanes of a group: each row's
// entries are dealt to the lanes in turn (a group reads whole 32-byte sectors of val), up to
// SROW of them in flight per lane, and the four rows' partials are exchanged so that lane l
// ends with the total of row row0 + l: three additions per lane for four rows, where a
// shuffle tree per row takes eight.  The products of a chunk end at the warp's longest row (a
// predicated-off FP64 instruction takes its 16 clocks of the pipe all the same).
template <class Col>
__device__ __forceinline__ double rowSums4(const int* rowptr, const int* col, const double* val, const double* x, int row0,
                                           int end, Col&& onEntry) {
    const int l = threadIdx.x & (SLANES - 1);
    if (row0 - (int)(threadIdx.x & 28) >= end) return 0.0;   // a warp without rows
    int ptr[SLANES + 1];
#pragma unroll
    for (int m = 0; m <= SLANES; m++) ptr[m] = __ldg(rowptr + min(row0 + m, end));
    double s[SLANES];
    double vv[SROW];
    int cc[SROW];
    auto load = [&](int k, int k1, double (&v)[SROW], int (&c)[SROW]) {
#pragma unroll
        for (int u = 0; u < SROW; u++) {
            const bool ok = k + u * SLANES < k1;
            c[u] = ok ? __ldg(col + k + u * SLANES) : -1;
            v[u] = ok ? __ldg(val + k + u * SLANES) : 0.0;
        }
    };
    load(ptr[0] + l, ptr[1], vv, cc);
#pragma unroll
    for (int m = 0; m < SLANES; m++) {
        s[m] = 0.0;
        const int k1 = ptr[m + 1];
        int k = ptr[m] + l;
        int most = __reduce_max_sync(0xffffffffu, (k1 - k + SLANES - 1) / SLANES);   // entries of the busiest lane
        while (true) {
            double g[SROW];
            int c[SROW];
#pragma unroll
            for (int u = 0; u < SROW; u++) { c[u] = cc[u]; g[u] = c[u] >= 0 ? x[c[u]] : 0.0; }
            double v[SROW];
#pragma unroll
            for (int u = 0; u < SROW; u++) v[u] = vv[u];
            // the next chunk's entries (the row's, or the next row's first) before the products
            const bool more = most > SROW;
            if (more) load(k + SROW * SLANES, k1, vv, cc);
            else if (m + 1 < SLANES) load(ptr[m + 1] + l, ptr[m + 2 < SLANES ? m + 2 : SLANES], vv, cc);
#pragma unroll
            for (int u = 0; u < SROW; u++) {
                if (u >= most) break;
                if (c[u] >= 0) {
                    onEntry(m, k + u * SLANES, c[u], v[u]);
                    s[m] += v[u] * g[u];
                }
            }
            if (!more) break;
            most -= SROW;
            k += SROW * SLANES;
        }
    }
    // lanes l and l ^ 2 trade two rows, then l and l ^ 1 one
    const bool h2 = l & 2, h1 = l & 1;
    const double a0 = __shfl_xor_sync(0xffffffffu, h2 ? s[0] : s[2], 2);
    const double a1 = __shfl_xor_sync(0xffffffffu, h2 ? s[1] : s[3], 2);
    const double b0 = (h2 ? s[2] : s[0]) + a0, b1 = (h2 ? s[3] : s[1]) + a1;
    const double c = __shfl_xor_sync(0xffffffffu, h1 ? b0 : b1, 1);
    return (h1 ? b1 : b0) + c;
}

// The whole solve in one cooperative launch.  Block b owns rows [b R, (b + 1) R), R = ceil(n /
// blocks), thread t the rows b R + t + m SBLK; r, p, Ap and the inverse diagonal of its rows
// stay in shared memory (vec != NULL: in global memory), z, which every block gathers, in
// global memory.  An iteration is
//   Ap = A z + beta Ap,  p = z + beta p,  alpha = r.z / p.Ap      (A p by linearity)
//   x += alpha p,  r -= alpha Ap,  z = M^-1 r,  r.z, r.r
// with two grid sums (about 3 us each: block tree, barrier, final sum and a division).  Measured
// at 108,000 rows of 30 entries: 22.2 us an iteration (of which about 8 us FP64 pipe; the
// 40 MB of matrix stay in the 129 MB L2), 11.2 us at 2,000 rows, where latencies bound it.
// Before, three launches an iteration, one thread summing the 256 block partials and a thread
// per row over the CSR entries: 84 us at 108,000 rows.
__global__ void __launch_bounds__(SBLK, 1) k_s_solve(int n, const int* rowptr, const int* col, const double* val,
                                                     const double* b, double* x, double* S, double tol, unsigned int maxIter,
                                                     int R, int inShared) {
    extern __shared__ __align__(16) double dyn[];
    __shared__ unsigned int badRow;
    __shared__ struct { double rz, bb, thr, alpha, beta; unsigned int done, it, breakdown, bad; } c;   // the block's scalars
    double* const z = S + OFF_Z;
    double* const scal = S + OFF_SCAL;
    unsigned int* const ctrl = (unsigned int*)(S + OFF_CTRL);
    const int r0 = blockIdx.x * R, r1 = min(n, r0 + R);
    const int cap = inShared ? R : SMAX;
    double* const vr = inShared ? dyn : S + OFF_VEC + r0;
    double* const vp = vr + cap;
    double* const vap = vp + cap;
    double* const vdi = vap + cap;
    GridBar g = {(unsigned long long*)(S + OFF_ARR), ctrl + C_ABORT, 0u};
    unsigned long long* const part = (unsigned long long*)(S + OFF_PART);
    const int active = min(SBLK, r1 - r0);
    const int t = threadIdx.x, l = t & (SLANES - 1);
    // rounds of SBLK rows: the same for every thread of the block (the row sums exchange lanes)
    const int rounds = (r1 - r0 + SBLK - 1) / SBLK;
    if (t == 0) badRow = 0u;
    __syncthreads();
    double v[3] = {0, 0, 0};
    for (int m = 0; m < rounds; m++) {
        const int q = m * SBLK + t, i = r0 + q;
        double diag[SLANES];   // this lane's diagonal entries of the group's rows (the last stored
        int at[SLANES];        // one, where a row stores several) and their places, -1: none
#pragma unroll
        for (int u = 0; u < SLANES; u++) { diag[u] = 0.0; at[u] = -1; }
        const int row0 = i - l;
        const double ax = rowSums4(rowptr, col, val, x, row0, r1, [&](int u, int k, int c, double a) {
            if (c == row0 + u) { diag[u] = a; at[u] = k; }
        });
        double di = 0.0;
#pragma unroll
        for (int u = 0; u < SLANES; u++) {   // the lane holding row u's diagonal gives it to lane u
            int k = max(at[u], __shfl_xor_sync(0xffffffffu, at[u], 1));
            k = max(k, __shfl_xor_sync(0xffffffffu, k, 2));
            const unsigned has = __ballot_sync(0xffffffffu, at[u] == k) & (0xfu << (t & 28));
            const double a = __shfl_sync(0xffffffffu, diag[u], __ffs(has) - 1);
            if (l == u && k >= 0) di = a;
        }
        if (i < r1) {
            // a row without a stored non-zero diagonal cannot be Jacobi-scaled: the lowest
            // such row is recorded (as UINT_MAX - row, so the maximum keeps the lowest)
            if (di != 0.0 && di == di) di = 1.0 / di;
            else { di = 0.0; atomicMax(&badRow, 0xFFFFFFFFu - (unsigned int)i); }
            const double bi = b[i], r = bi - ax, zi = r * di;
            vdi[q] = di; vr[q] = r; z[i] = zi;
            v[0] += r * zi; v[1] += r * r; v[2] += bi * bi;
        }
    }
    __syncthreads();
    if (t == 0 && badRow) atomicMax(ctrl + C_BADROW, badRow);
    if (!gridTotal<3>(v, g, part, active, [&](const double* d) {
            c.rz = d[0];
            c.bb = d[2];
            c.thr = fmax(tol * tol * d[2], 2.2250738585072014e-308);
            c.breakdown = !(d[0] == d[0]) || !(d[1] == d[1]);
            c.done = (d[2] == 0.0 || d[1] < c.thr || c.breakdown) ? 1u : 0u;
            c.it = 0u;
            c.bad = *(volatile unsigned int*)(ctrl + C_BADROW);
        }))
        return;
    // a malformed system is rejected by the host with x untouched; a zero right-hand side has
    // the solution x = 0 (as Eigen's CG returns)
    if (c.bad || c.bb == 0.0) {
        if (!c.bad)
            for (int q = t; q < r1 - r0; q += SBLK) x[r0 + q] = 0.0;
        if (blockIdx.x == 0 && t == 0) { scal[SC_BB] = c.bb; scal[SC_RR0] = 0.0; ctrl[C_DONE] = 1u; }
        return;
    }
    while (!c.done && c.it < maxIter) {
        const bool first = c.it == 0u;
        double a1[1] = {0};
        for (int m = 0; m < rounds; m++) {
            const int q = m * SBLK + t, i = r0 + q;
            const double az = rowSums4(rowptr, col, val, z, i - l, r1, [](int, int, int, double) {});
            if (i < r1) {
                const double zi = z[i];
                const double ap = first ? az : az + c.beta * vap[q], p = first ? zi : zi + c.beta * vp[q];
                vap[q] = ap; vp[q] = p;
                a1[0] += p * ap;
            }
        }
        if (!gridTotal<1>(a1, g, part, active, [&](const double* d) { c.alpha = c.rz / d[0]; })) return;
        const double alpha = c.alpha;
        double a2[2] = {0, 0};
        for (int q = t; q < r1 - r0; q += SBLK) {
            x[r0 + q] += alpha * vp[q];
            const double r = vr[q] - alpha * vap[q], zi = r * vdi[q];
            vr[q] = r; z[r0 + q] = zi;
            a2[0] += r * zi; a2[1] += r * r;
        }
        if (!gridTotal<2>(a2, g, part, active, [&](const double* d) {
                c.it += 1u;
                c.beta = d[0] / c.rz;
                c.rz = d[0];
                if (d[1] < c.thr) c.done = 1u;
                else if (c.it >= maxIter) c.done = 2u;   // stopped at the iteration cap
                if (!(d[1] == d[1])) { c.done = 1u; c.breakdown = 1u; }
            }))
            return;
    }
    // true residual (x of every block is complete at the last sum)
    double a1[1] = {0};
    for (int m = 0; m < rounds; m++) {
        const int q = m * SBLK + t, i = r0 + q;
        const double ax = rowSums4(rowptr, col, val, x, i - l, r1, [](int, int, int, double) {});
        if (i < r1) {
            const double r = b[i] - ax;
            a1[0] += r * r;
        }
    }
    if (!gridTotal<1>(a1, g, part, active, [&](const double* d) {
            if (blockIdx.x) return;
            scal[SC_BB] = c.bb; scal[SC_RR0] = d[0];
            ctrl[C_DONE] = c.done; ctrl[C_ITERS] = c.it; ctrl[C_BREAK] = c.breakdown;
        }))
        return;
}

// One call at a time on a device: the scratch is shared, and the solve's blocks wait on one
// another through it.
std::mutex g_callMu[256];
std::mutex g_mu;
double* g_addr[256] = {nullptr};
std::string g_msg;

// Device address of the scratch array for the current device (looked up once per device).
int scratchFor(double** out, int* devOut) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) { g_msg = "no current CUDA device"; return MPSGPU_ERR_NOGPU; }
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_addr[dev]) {
        double* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void**)&p, g_pcgScratch);
        if (e != cudaSuccess || !p) {
            g_msg = std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e);
            return MPSGPU_ERR_CUDA;
        }
        g_addr[dev] = p;
    }
    *out = g_addr[dev];
    *devOut = dev;
    return 0;
}

}  // namespace

extern "C" int mpsgpu_pcg_solve_static(int n, const int* rowptr, const int* col, const double* val,
                                       const double* b, double* x, double tol, int max_iter, void* stream,
                                       int* iters, double* relres) {
    if (n <= 0 || n > SMAX) {
        g_msg = "mpsgpu_pcg_solve_static: " + std::to_string(n) + " rows outside 1.." + std::to_string(SMAX) +
                " (the static scratch holds MPSGPU_STATIC_MAX_ROWS rows)";
        return MPSGPU_ERR_ARG;
    }
    if (!rowptr || !col || !val || !b || !x || !(tol > 0) || max_iter <= 0) {
        g_msg = "mpsgpu_pcg_solve_static: bad argument";
        return MPSGPU_ERR_ARG;
    }
    double* S = nullptr;
    int dev = 0, sms = 0;
    int e = scratchFor(&S, &dev);
    if (e) return e;
    cudaStream_t s = (cudaStream_t)stream;
    auto fail = [](const char* what, cudaError_t err) {
        g_msg = std::string("mpsgpu_pcg_solve_static: ") + what + ": " + cudaGetErrorString(err);
        return MPSGPU_ERR_CUDA;
    };
    cudaError_t ce = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (ce != cudaSuccess) return fail("device", ce);
    std::lock_guard<std::mutex> call(g_callMu[dev]);
    // one block per SM, fewer where a block would own under 64 rows (its 16 row groups per
    // round would idle and every further block lengthens the grid sums)
    int nb = (n + 63) / 64;
    if (nb > sms) nb = sms;
    if (nb > SBLOCKS) nb = SBLOCKS;
    int R = (n + nb - 1) / nb, inShared = 1;
    nb = (n + R - 1) / R;
    size_t dyn = sizeof(double) * 4 * (size_t)R;
    if (dyn > 160 * 1024) { dyn = 0; inShared = 0; }   // few SMs: the vectors go to the scratch
    if (dyn && (ce = cudaFuncSetAttribute(k_s_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn)) != cudaSuccess)
        return fail("shared memory", ce);
    // the array keeps the previous call's contents: reset the scalars, control words and arrivals
    const size_t headBytes = sizeof(double) * (16 + 4);
    ce = cudaMemsetAsync(S + OFF_SCAL, 0, sizeof(double) * (OFF_PART - OFF_SCAL), s);
    if (ce != cudaSuccess) return fail("clearing the control words", ce);
    unsigned int mi = (unsigned int)max_iter;
    void* args[] = {&n, &rowptr, &col, &val, &b, &x, &S, &tol, &mi, &R, &inShared};
    if ((ce = cudaLaunchCooperativeKernel((const void*)k_s_solve, nb, SBLK, args, dyn, s)) != cudaSuccess)
        return fail("launch", ce);
    double head[20];
    if ((ce = cudaMemcpyAsync(head, S + OFF_SCAL, headBytes, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (ce = cudaStreamSynchronize(s)) != cudaSuccess)
        return fail("solve", ce);
    unsigned int ctrl[8];
    std::memcpy(ctrl, head + 16, sizeof(ctrl));
    if (ctrl[C_ABORT]) { g_msg = "mpsgpu_pcg_solve_static: a grid wait ran out"; return MPSGPU_ERR_CUDA; }
    if (ctrl[C_BADROW]) {
        g_msg = "mpsgpu_pcg_solve_static: row " + std::to_string(0xFFFFFFFFu - ctrl[C_BADROW]) +
                " has no stored non-zero diagonal entry (Jacobi preconditioning needs one in every row)";
        return MPSGPU_ERR_ARG;
    }
    if (iters) *iters = (int)ctrl[C_ITERS];
    if (head[SC_BB] == 0.0) {
        if (relres) *relres = 0.0;
        return 0;
    }
    if (relres) *relres = std::sqrt(head[SC_RR0] / head[SC_BB]);
    if (ctrl[C_BREAK] || ctrl[C_DONE] != 1u) { g_msg = "mpsgpu_pcg_solve_static: did not reach the tolerance"; return MPSGPU_ERR_NOT_CONVERGED; }
    return 0;
}

extern "C" const char* mpsgpu_pcg_static_error(void) { return g_msg.c_str(); }
