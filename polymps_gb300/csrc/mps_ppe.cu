// mps_ppe.cu — pressure Poisson equation on sm_103a: assembly and solvers.
//
// Assembly replaces the serial Eigen triplet loop of MpsPressure::solvePressurePoissonPnd
// (src/MpsPressure.cpp:169-286): one thread per row walks its ELL neighbour row and writes
// the off-diagonal entries (j inner, not dummy) straight into an ELL matrix
// (val/col at ellBase(i) + k ellStride, coalesced across a warp), the diagonal and the right-hand side.
//
// The plain solver replaces Eigen's ConjugateGradient<..., Lower|Upper> with its default
// diagonal preconditioner (src/MpsPressure.cpp:424-445): Jacobi-PCG in FP64 warm-started
// from the previous unclamped solution, stopping when ||r||^2 < tol^2 ||b||^2.  Per
// iteration three grid-stride kernels (SpMV + p.Ap, x/r/z update + r.z and r.r,
// p update); the scalar reductions are deterministic (per-block partials, the last block
// to finish sums them in block order) and the solver state stays on the device: the host
// only polls the "done" word every few iterations.
//
// The mixed solver keeps FP64 for the iterative-refinement residual r = b - Ax, its norm
// and all dot products, and runs the inner CG on FP32 matrix values and vectors.
#include "mps_df.cuh"
#include "mps_internal.h"
#include <algorithm>
#include "mps_bulk.cuh"
#include "mps_grid.cuh"
#include "mps_lanes.cuh"

#define PBLK 256

// solver scalars in B.scal[]
enum { S_RZ = 0, S_RR, S_BB, S_ALPHA, S_BETA, S_PAP, S_THR, S_RZNEW, S_SCALE, S_INV, S_SQRT, S_ETA2, S_RR0,
       S_RHO, S_RHOOLD, S_OMEGA, S_R0N2, S_COUNT };

// ------------------------------------------------------------------ assembly
// The row of particle i by L lanes.  Dummy-wall neighbours (their hydrostatic source term, 12
// FP64 operations) are left to a second walk over the few there are: in the loop, every entry
// of every particle paid for them (864k particles without any: 596 -> 172 us).
template <int L>
__global__ void __launch_bounds__(128) k_ppe_assemble(Dev d, PpeBuffers B) {
    const int i = laneRow<L>(), l = laneOf<L>();
    if (i >= liveN(d)) return;
    const MpsParams& P = d.P;
    if (l == 0) B.x[i] = d.pressPPE[i];   // the start of a solve from the previous solution
    const int bci = d.bc[i];
    if (bci == P.other || bci == P.surface) {
        if (l == 0) { B.diag[i] = 1.0; B.rowLen[i] = 0; B.b[i] = 0.0; B.mfMask[i] = maskNone(); }
        warpCount(d.counters + 1, 0u);
        return;
    }
    double sum = 0.0, src = 0.0;
    Mask mm = maskNone(), dm = maskNone();
    const double* wLc = d.cwL ? d.cwL : d.cw;
    const Mask mL = d.maskL[i];
    const size_t base = ellBase(B, i);
    int len = 0;
    if (L > 1) {   // the matrix entries of the whole row first: an entry's place is its rank
        forMaskLane<L>(d, i, mL, l, [&](int j, size_t, int k) {
            if (d.type[j] != P.dummyWall && d.bc[j] == P.inner) maskSet(mm, k);
        });
        mm = laneOr<L>(mm);
        len = maskCount(mm);
    }
    forMaskLane<L>(d, i, mL, l, [&](int j, size_t e, int k) {
        if (d.type[j] == P.dummyWall) { maskSet(dm, k); return; }
        const double mij = wLc[e] * P.coeffPPE;
        sum -= mij;
        if (d.bc[j] != P.inner) return;
        int at;
        if (L > 1) at = maskRank(mm, k);
        else { at = len++; maskSet(mm, k); }
        B.val[base + (size_t)at * B.ellStride] = mij;
        B.col[base + (size_t)at * B.ellStride] = j;
    });
    if (dm.lo | dm.hi) {
        const dvec4 pi = d.pos[i];
        forBits(d.nbr + i, d.N0, dm, [&](int j, int k) {
            const dvec4 pj = d.pos[j];
            const double v0 = pj.x - pi.x, v1 = pj.y - pi.y, v2 = pj.z - pi.z;
            const double pgh = P.DNS_FL1 * (v0 * P.gravity[0] + v1 * P.gravity[1] + v2 * P.gravity[2]) *
                               wLc[(size_t)k * d.N0 + i];
            src -= P.coeffPPE * pgh;
        });
    }
    sum = laneSum<L>(sum);
    src = laneSum<L>(src);
    if (l == 0) {
        const double rho = P.DNS_FL1;
        sum -= P.alphaCompressibility * rho / (P.timeStep * P.timeStep);
        B.diag[i] = sum;
        B.rowLen[i] = len;
        B.mfMask[i] = mm;
        B.b[i] = src + ppeSource(d, i, rho);
    }
    warpCount(d.counters + 1, l == 0 ? (unsigned)len : 0u);
}
void launchPpeAssemble(const Dev& d, const PpeBuffers& B, cudaStream_t s) {
    cudaMemsetAsync(d.counters + 1, 0, sizeof(unsigned long long), s);
#define LAUNCH(L) k_ppe_assemble<L><<<gridFor(d.N0 * L, 128), 128, 0, s>>>(d, B)
    MPS_FOR_LANES(d.N0, LAUNCH);
#undef LAUNCH
}

// press = max(x, 0) (setZeroOnNegativePressure, src/MpsPressure.cpp:471-476); x is kept
// unclamped in pressPPE as the next warm start.
__global__ void k_ppe_copy_back(Dev d, PpeBuffers B) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    double x = B.x[i];
    d.pressPPEprev2[i] = d.pressPPEprev[i];
    d.pressPPEprev[i] = d.pressPPE[i];
    d.pressPPE[i] = x;
    d.source[i] = B.b[i];
    d.press[i] = x < 0.0 ? 0.0 : x;
}
// Warm start by extrapolation in time of the unclamped solutions on the rows of the new
// system that carry an equation (zero on the identity rows): linear x0 = 2 p_n - p_{n-1}
// or quadratic x0 = 3 p_n - 3 p_{n-1} + p_{n-2}.
__global__ void k_warm_extrap(Dev d, PpeBuffers B, int quad) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    double p = d.pressPPE[i], q = d.pressPPEprev[i];
    double x = quad ? 3.0 * (p - q) + d.pressPPEprev2[i] : (p + p) - q;
    B.x[i] = (d.bc[i] == d.P.inner) ? x : 0.0;
}
void launchWarmExtrapolate(const Dev& d, const PpeBuffers& B, cudaStream_t s, bool quadratic) {
    k_warm_extrap<<<gridFor(d.N0, 256), 256, 0, s>>>(d, B, quadratic ? 1 : 0);
}
void launchPpeCopyBack(const Dev& d, const PpeBuffers& B, cudaStream_t s) {
    k_ppe_copy_back<<<gridFor(d.N0, 256), 256, 0, s>>>(d, B);
}

// ------------------------------------------------------------------ reductions
// Block-wide sum of NV doubles; the last block to arrive sums the per-block partials in
// block order (deterministic) and calls fin(tot) with thread 0.
template <int NV>
__device__ __forceinline__ void blockSum(double (&v)[NV], double* sm) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    }
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; q++) sm[q * 32 + w] = v[q];
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            double x = (lane < nw) ? sm[q * 32 + lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            v[q] = x;
        }
    }
    __syncthreads();
}

template <int NV, class Fin>
__device__ __forceinline__ void gridSum(double (&v)[NV], const PpeBuffers& B, Fin fin) {
    __shared__ double sm[NV * 32];
    __shared__ bool last;
    blockSum<NV>(v, sm);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) B.partials[q * gridDim.x + blockIdx.x] = v[q];
        __threadfence();
        unsigned int t = atomicInc(B.counter, gridDim.x - 1);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
        double s = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
            s += ((volatile double*)B.partials)[q * gridDim.x + b];
        acc[q] = s;
    }
    blockSum<NV>(acc, sm);
    if (threadIdx.x == 0) fin(acc);
}

// ------------------------------------------------------------------ ELL rows (ellRow: mps_common.cuh)
__device__ __forceinline__ double spmvRow(const PpeBuffers& B, const double* x, int i) {
    return ellRow<double, true>(B.diag, B.val, B.col, x, i, __ldg(B.rowLen + i), ellBase(B, i), B.ellStride);
}

// r = b - A x, z = r / diag, p = z; sums r.z, r.r, b.b
__global__ void __launch_bounds__(PBLK) k_cg_init(Dev d, PpeBuffers B, double tol) {
    int n = liveN(d);
    double v[3] = {0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double r = B.b[i] - spmvRow(B, B.x, i);
        double z = r / B.diag[i];
        B.r[i] = r; B.z[i] = z; B.p[i] = z;
        v[0] += r * z; v[1] += r * r; v[2] += B.b[i] * B.b[i];
    }
    gridSum<3>(v, B, [&](double* t) {
        B.scal[S_RZ] = t[0]; B.scal[S_RR] = t[1]; B.scal[S_BB] = t[2];
        double thr = tol * tol * t[2];
        if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
        B.scal[S_THR] = thr;
        B.scal[S_SCALE] = sqrt(t[1] / (t[2] > 0 ? t[2] : 1.0));   // initial relative residual
        B.flag[0] = (t[2] == 0.0 || t[1] < thr) ? 1 : 0;
        B.flag[1] = 0;
        if (!(t[0] == t[0]) || !(t[1] == t[1])) { B.flag[0] = 1; B.flag[2] = 1; }
    });
}
// Ap = A p; sum p.Ap -> alpha
__global__ void __launch_bounds__(PBLK) k_cg_spmv(Dev d, PpeBuffers B) {
    if (*(volatile int*)B.flag) return;
    int n = liveN(d);
    double v[1] = {0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double ap = spmvRow(B, B.p, i);
        B.Ap[i] = ap;
        v[0] += B.p[i] * ap;
    }
    gridSum<1>(v, B, [&](double* t) { B.scal[S_PAP] = t[0]; B.scal[S_ALPHA] = B.scal[S_RZ] / t[0]; });
}
// x += alpha p; r -= alpha Ap; z = r/diag; sums r.z, r.r -> beta, convergence
__global__ void __launch_bounds__(PBLK) k_cg_update(Dev d, PpeBuffers B) {
    if (*(volatile int*)B.flag) return;
    int n = liveN(d);
    double alpha = B.scal[S_ALPHA];
    double v[2] = {0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double p = B.p[i];
        B.x[i] += alpha * p;
        double r = B.r[i] - alpha * B.Ap[i];
        double z = r / B.diag[i];
        B.r[i] = r; B.z[i] = z;
        v[0] += r * z; v[1] += r * r;
    }
    gridSum<2>(v, B, [&](double* t) {
        B.flag[1] += 1;
        B.scal[S_RR] = t[1];
        B.scal[S_BETA] = t[0] / B.scal[S_RZ];
        B.scal[S_RZ] = t[0];
        if (t[1] < B.scal[S_THR]) B.flag[0] = 1;
        if (!(t[1] == t[1])) { B.flag[0] = 1; B.flag[2] = 1; }
    });
}
// p = z + beta p
__global__ void __launch_bounds__(PBLK) k_cg_p(Dev d, PpeBuffers B) {
    if (*(volatile int*)B.flag) return;
    int n = liveN(d);
    double beta = B.scal[S_BETA];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        B.p[i] = B.z[i] + beta * B.p[i];
}
// true residual ||b - A x||^2 (FP64) into scal[S_RR]
__global__ void __launch_bounds__(PBLK) k_true_residual(Dev d, PpeBuffers B) {
    int n = liveN(d);
    double v[1] = {0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double r = B.b[i] - spmvRow(B, B.x, i);
        B.r[i] = r;
        v[0] += r * r;
    }
    gridSum<1>(v, B, [&](double* t) { B.scal[S_RR] = t[0]; });
}

static int pollFlags(const PpeBuffers& B, cudaStream_t s, int* hostFlags) {
    if (cudaMemcpyAsync(hostFlags, B.flag, 3 * sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    return 0;
}

int ppeSolvePlain(const Dev& d, const PpeBuffers& B, double tol, int maxIter, cudaStream_t s,
                  int* iters, double* relres, double* relres0, Prof* prof) {
    int nb = B.nblocks;
    static thread_local int hf[4];
    bool pr = prof && prof->on;
    cudaMemsetAsync(B.flag, 0, 4 * sizeof(int), s);
    if (pr) prof->begin(PROF_PPE_OTHER, s);
    k_cg_init<<<nb, PBLK, 0, s>>>(d, B, tol);
    if (pr) prof->end(s);
    countLaunch(1);
    const int batch = 8;
    int launched = 0;
    while (true) {
        for (int k = 0; k < batch; k++) {
            if (pr) prof->begin(PROF_PPE_SPMV, s);
            k_cg_spmv<<<nb, PBLK, 0, s>>>(d, B);
            if (pr) { prof->end(s); prof->begin(PROF_PPE_VECTOR, s); }
            k_cg_update<<<nb, PBLK, 0, s>>>(d, B);
            k_cg_p<<<nb, PBLK, 0, s>>>(d, B);
            if (pr) prof->end(s);
        }
        countLaunch(3 * batch);
        launched += batch;
        if (pollFlags(B, s, hf)) return MPSGPU_ERR_CUDA;
        if (hf[0] || launched >= maxIter) break;
    }
    double sc[S_COUNT];
    countLaunch(1);
    k_true_residual<<<nb, PBLK, 0, s>>>(d, B);
    cudaMemcpyAsync(sc, B.scal, sizeof(sc), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return MPSGPU_ERR_CUDA;
    *iters = hf[1];
    double bb = sc[S_BB] > 0 ? sc[S_BB] : 1.0;
    *relres = (sc[S_BB] > 0) ? sqrt(sc[S_RR] / bb) : 0.0;
    *relres0 = sc[S_SCALE];
    if (hf[2]) return MPSGPU_ERR_NOT_CONVERGED;
    if (!hf[0]) return MPSGPU_ERR_NOT_CONVERGED;
    return 0;
}

// ------------------------------------------------------------------ mixed FP32/FP64
// FP32 copies of the matrix values and the Jacobi inverse diagonal
__global__ void k_mixed_prepare(Dev d, PpeBuffers B) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    int len = B.rowLen[i];
    const size_t base = ellBase(B, i);
    for (int k = 0; k < len; k++) {
        size_t e = base + (size_t)k * B.ellStride;
        B.valf[e] = (float)B.val[e];
    }
    B.diagf[i] = (float)B.diag[i];
    B.diagInvf[i] = (float)(1.0 / B.diag[i]);
}
void launchMixedPrepare(const Dev& d, const PpeBuffers& B, cudaStream_t s) {
    k_mixed_prepare<<<gridFor(d.N0, 256), 256, 0, s>>>(d, B);
}
// FP64 residual r = b - A x (FP64 values), sums r.r (and b.b on the first call)
__global__ void __launch_bounds__(PBLK) k_mx_residual(Dev d, PpeBuffers B, int first, double tol) {
    int n = liveN(d);
    double v[2] = {0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double r = B.b[i] - spmvRow(B, B.x, i);
        B.r[i] = r;
        v[0] += r * r;
        if (first) v[1] += B.b[i] * B.b[i];
    }
    gridSum<2>(v, B, [&](double* t) {
        B.scal[S_RR] = t[0];
        if (first) {
            B.scal[S_BB] = t[1];
            double thr = tol * tol * t[1];
            if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
            B.scal[S_THR] = thr;
            B.scal[S_SCALE] = sqrt(t[0] / (t[1] > 0 ? t[1] : 1.0));
        }
        B.flag[0] = (B.scal[S_BB] == 0.0 || t[0] < B.scal[S_THR]) ? 1 : 0;
        if (!(t[0] == t[0])) { B.flag[0] = 1; B.flag[2] = 1; }
    });
}
// inner start: rf = r / ||r||, d = 0, z = M rf, p = z; r.z (FP64 accumulate)
__global__ void __launch_bounds__(PBLK) k_mx_inner_init(Dev d, PpeBuffers B) {
    int n = liveN(d);
    double inv = 1.0 / sqrt(B.scal[S_RR]);
    double v[1] = {0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float r = (float)(B.r[i] * inv);
        float z = r * B.diagInvf[i];
        B.rf[i] = r; B.zf[i] = z; B.pf[i] = z; B.xf[i] = 0.f;
        v[0] += (double)r * (double)z;
    }
    gridSum<1>(v, B, [&](double* t) { B.scal[S_RZ] = t[0]; B.flag[3] = 0; });
}
__device__ __forceinline__ float spmvRowF(const PpeBuffers& B, const float* x, int i) {
    return ellRow<float, true>(B.diagf, B.valf, B.col, x, i, __ldg(B.rowLen + i), ellBase(B, i), B.ellStride);
}
__global__ void __launch_bounds__(PBLK) k_mx_spmv(Dev d, PpeBuffers B) {
    if (*(volatile int*)(B.flag + 3)) return;
    int n = liveN(d);
    double v[1] = {0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float ap = spmvRowF(B, B.pf, i);
        B.Apf[i] = ap;
        v[0] += (double)B.pf[i] * (double)ap;
    }
    gridSum<1>(v, B, [&](double* t) { B.scal[S_ALPHA] = B.scal[S_RZ] / t[0]; });
}
// inner tolerance eta on the normalised residual (||rf_0|| = 1)
__global__ void __launch_bounds__(PBLK) k_mx_update(Dev d, PpeBuffers B, double eta2) {
    if (*(volatile int*)(B.flag + 3)) return;
    int n = liveN(d);
    float alpha = (float)B.scal[S_ALPHA];
    double v[2] = {0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float p = B.pf[i];
        B.xf[i] += alpha * p;
        float r = B.rf[i] - alpha * B.Apf[i];
        float z = r * B.diagInvf[i];
        B.rf[i] = r; B.zf[i] = z;
        v[0] += (double)r * (double)z; v[1] += (double)r * (double)r;
    }
    gridSum<2>(v, B, [&](double* t) {
        B.flag[1] += 1;
        B.scal[S_BETA] = t[0] / B.scal[S_RZ];
        B.scal[S_RZ] = t[0];
        if (t[1] < eta2 || !(t[1] == t[1])) B.flag[3] = 1;
    });
}
__global__ void __launch_bounds__(PBLK) k_mx_p(Dev d, PpeBuffers B) {
    if (*(volatile int*)(B.flag + 3)) return;
    int n = liveN(d);
    float beta = (float)B.scal[S_BETA];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        B.pf[i] = B.zf[i] + beta * B.pf[i];
}
// x += ||r|| * d  (FP64)
__global__ void k_mx_correct(Dev d, PpeBuffers B) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= liveN(d)) return;
    double sc = sqrt(B.scal[S_RR]);
    B.x[i] += sc * (double)B.xf[i];
}

int ppeSolveMixed(const Dev& d, const PpeBuffers& B, double tol, int maxIter, cudaStream_t s,
                  int* iters, int* refinements, double* relres, double* relres0, Prof* prof) {
    int nb = B.nblocks;
    static thread_local int hf[4];
    bool pr = prof && prof->on;
    cudaMemsetAsync(B.flag, 0, 4 * sizeof(int), s);
    if (pr) prof->begin(PROF_PPE_OTHER, s);
    k_mixed_prepare<<<gridFor(d.N0, 256), 256, 0, s>>>(d, B);
    k_mx_residual<<<nb, PBLK, 0, s>>>(d, B, 1, tol);
    if (pr) prof->end(s);
    countLaunch(2);
    int refine = 0, total = 0;
    const double eta = 2e-4;   // inner relative tolerance (FP32 CG stagnates near 1e-6)
    const int batch = 8;
    while (true) {
        if (pollFlags(B, s, hf)) return MPSGPU_ERR_CUDA;
        if (hf[0] || total >= maxIter) break;
        k_mx_inner_init<<<nb, PBLK, 0, s>>>(d, B);
        countLaunch(1);
        int inner = 0;
        while (true) {
            for (int k = 0; k < batch; k++) {
                if (pr) prof->begin(PROF_PPE_SPMV, s);
                k_mx_spmv<<<nb, PBLK, 0, s>>>(d, B);
                if (pr) { prof->end(s); prof->begin(PROF_PPE_VECTOR, s); }
                k_mx_update<<<nb, PBLK, 0, s>>>(d, B, eta * eta);
                k_mx_p<<<nb, PBLK, 0, s>>>(d, B);
                if (pr) prof->end(s);
            }
            countLaunch(3 * batch);
            inner += batch;
            int f4[4];
            if (cudaMemcpyAsync(f4, B.flag, 4 * sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return MPSGPU_ERR_CUDA;
            if (cudaStreamSynchronize(s) != cudaSuccess) return MPSGPU_ERR_CUDA;
            if (f4[3] || total + inner >= maxIter || inner >= 400) break;
        }
        total += inner;
        if (pr) prof->begin(PROF_PPE_OTHER, s);
        k_mx_correct<<<gridFor(d.N0, 256), 256, 0, s>>>(d, B);
        k_mx_residual<<<nb, PBLK, 0, s>>>(d, B, 0, tol);
        if (pr) prof->end(s);
        countLaunch(2);
        refine++;
        if (refine > 20) break;
    }
    double sc[S_COUNT];
    cudaMemcpyAsync(sc, B.scal, sizeof(sc), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return MPSGPU_ERR_CUDA;
    *iters = hf[1];
    *refinements = refine;
    double bb = sc[S_BB] > 0 ? sc[S_BB] : 1.0;
    *relres = (sc[S_BB] > 0) ? sqrt(sc[S_RR] / bb) : 0.0;
    *relres0 = sc[S_SCALE];
    if (hf[2] || !hf[0]) return MPSGPU_ERR_NOT_CONVERGED;
    return 0;
}

// ------------------------------------------------------------------ persistent solvers
// The whole solve in one cooperative launch (every block co-resident): no host polling,
// no per-iteration launches.  Each CG iteration is two grid-wide reductions in the form
//   Ap = A z + beta Ap,  p = z + beta p            (one SpMV, on z: A p follows by linearity)
//   x += alpha p, r -= alpha Ap, z = M^-1 r
// so the only vector every block gathers (z) is complete at the reduction before it.
// A reduction is one barrier: every block stores its partial sums, adds one to the
// arrival counter (release) and polls it until it reaches the generation's target; then
// every block sums all partials in block order and derives the solver's
// scalars itself.  Identical inputs in identical order give every block identical
// scalars, so no block has to publish them and release the others.  The scalars and flags
// live in shared memory per block; block 0 stores its copy for the host at the end.  Waits are
// bounded: a block that waits longer than GRID_SPIN polls sets the abort word and every
// block returns.
// Block sizes: one block per SM (1024 threads for the mixed solvers at <= 64 registers,
// 768 for the FP64 solvers at <= 80), so a reduction reads 152 partials per value
// instead of 608 (every block reads them all: measured 12 -> 7 us per reduction); the
// staged-tile operator keeps 256-thread blocks (its tiles are one row per thread).
#define QB 256
#define QBX 1024
#define QBC 768
// barrier words, each on its own 128-byte line (the arrival counter is 64-bit and only
// grows within a launch; it is zeroed before each launch): arrivals, unused, abort
#define QB_ARR 0
#define QB_ABT 64
#define QB_WORDS 96

__device__ __forceinline__ double vd(const double* p) { return *(volatile const double*)p; }
__device__ __forceinline__ int vi(const int* p) { return *(volatile const int*)p; }

struct QCtl {
    unsigned int gen;
};
// block-local solver scalars and flags
struct QLocal {
    double scal[32];
    int flag[8];
    float scalf[4];   // FP32 copies of the inner-CG step scalars (SF_*), formed once by thread 0
};
#define SF_ALPHA 0
#define SF_BETA 1
__device__ __forceinline__ void qInit(QLocal& L) {
    for (int t = threadIdx.x; t < 32; t += blockDim.x) L.scal[t] = 0.0;
    for (int t = threadIdx.x; t < 8; t += blockDim.x) L.flag[t] = 0;
    for (int t = threadIdx.x; t < 4; t += blockDim.x) L.scalf[t] = 0.f;
    __syncthreads();
}
__device__ __forceinline__ float vf(const float* p) { return *(volatile const float*)p; }
// block 0's scalars and flags to the global words the host reads
__device__ __forceinline__ void qStore(const PpeBuffers& B, const QLocal& L) {
    __syncthreads();
    if (blockIdx.x == 0) {
        for (int t = threadIdx.x; t < 32; t += blockDim.x) B.scal[t] = L.scal[t];
        for (int t = threadIdx.x; t < 8; t += blockDim.x) B.flag[t] = L.flag[t];
    }
}

__device__ __forceinline__ GridBar qBar(const PpeBuffers& B, const QCtl& c) {
    return {reinterpret_cast<unsigned long long*>(B.bar + QB_ARR), B.bar + QB_ABT, c.gen};
}
// Grid barrier: all writes of the block before it are visible to every block after it.
__device__ __forceinline__ bool qBarrier(const PpeBuffers& B, QCtl& c) {
    GridBar g = qBar(B, c);
    c.gen++;
    return gridBarrier(g);
}
// The grid's sum of NV (<= 4) values from the blocks' partials pv (thread 0's), by warp 0 of
// every block in the same order: got(word) turns a partial's word into a T, which add
// sums; fin(tot) runs on thread 0 with the totals, and its writes to the block-local scalars
// are visible to the block's threads on return.  The block has passed a __syncthreads since
// its last global write.  The partials of consecutive reductions alternate between two
// buffers: a block can be at most one reduction ahead of the slowest block's reads.
template <int NV, class T, class Got, class Xor, class Fin>
__device__ __forceinline__ bool qCollect(const unsigned long long (&pv)[NV], const PpeBuffers& B, QCtl& c, Got&& got,
                                         Xor&& xorLane, Fin&& fin) {
    c.gen++;
    int ok = 1;
    if (threadIdx.x < 32) {
        GridBar g = qBar(B, c);
        unsigned long long* const set = reinterpret_cast<unsigned long long*>(B.partials) + (size_t)(c.gen & 1u) * 4u * gridDim.x;
        if (threadIdx.x == 0)
#pragma unroll
            for (int q = 0; q < NV; q++)
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(set + q * gridDim.x + blockIdx.x), "l"(pv[q]) : "memory");
        ok = gridWaitWarp0(g);
        if (ok) {
            T tot[NV];
#pragma unroll
            for (int q = 0; q < NV; q++) tot[q] = got(0ull);
            // five partials of a lane (160 blocks) in flight at a time
            for (unsigned b0 = 0; b0 < gridDim.x; b0 += 160) {
                unsigned long long w[NV][5];
#pragma unroll
                for (int q = 0; q < NV; q++)
#pragma unroll
                    for (int m = 0; m < 5; m++) {
                        const unsigned b = b0 + threadIdx.x + 32 * m;
                        w[q][m] = b < gridDim.x ? ldRelaxed(set + q * gridDim.x + b) : 0ull;
                    }
#pragma unroll
                for (int q = 0; q < NV; q++)
                    tot[q] += ((got(w[q][0]) + got(w[q][1])) + (got(w[q][2]) + got(w[q][3]))) + got(w[q][4]);
            }
#pragma unroll
            for (int q = 0; q < NV; q++)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) tot[q] += xorLane(tot[q], o);
            if (threadIdx.x == 0) fin(tot);
        }
    }
    return __syncthreads_and(ok) != 0;
}
// Grid sum of NV FP64 values per thread.
template <int NV, class Fin>
__device__ __forceinline__ bool qSum(double (&v)[NV], const PpeBuffers& B, QCtl& c, Fin fin) {
    __shared__ double sm[NV * 32];
    blockSum<NV>(v, sm);
    unsigned long long pv[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) pv[q] = (unsigned long long)__double_as_longlong(v[q]);
    return qCollect<NV, double>(
        pv, B, c, [](unsigned long long w) { return __longlong_as_double((long long)w); },
        [](double x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); }, fin);
}
// The same with float-float per-thread partials (FP32 vectors), reduced in float-float all
// the way: the warps' shuffle trees, the block's sum of its warps, the block partials (two
// floats in the same partial slots) and the final sum over the blocks; fin takes the
// float-float totals.  In FP64 the shuffle trees of every warp and the final sum ran on the
// FP64 pipe (1/64 of the FP32 rate) between the last arrival and the release of every barrier.
__device__ __forceinline__ df shflXorDF(df a, int o) {
    return {__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)};
}
template <int NV, class Fin>
__device__ __forceinline__ bool qSumF2(df (&a)[NV], const PpeBuffers& B, QCtl& c, Fin fin, bool any = true) {
    __shared__ float2 sm[NV * 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        if (any) {   // a warp without rows keeps its zeros: its trees would take the others' issue slots
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a[q] += shflXorDF(a[q], o);
        }
        if (lane == 0) sm[q * 32 + w] = make_float2(a[q].h, a[q].l);
    }
    __syncthreads();
    unsigned long long pv[NV];
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const float2 x = (lane < nw) ? sm[q * 32 + lane] : make_float2(0.f, 0.f);
            df s = {x.x, x.y};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += shflXorDF(s, o);
            pv[q] = (unsigned long long)__float_as_uint(s.h) | ((unsigned long long)__float_as_uint(s.l) << 32);
        }
    }
    return qCollect<NV, df>(
        pv, B, c, [](unsigned long long u) { return df{__uint_as_float((unsigned)u), __uint_as_float((unsigned)(u >> 32))}; },
        [](df x, int o) { return shflXorDF(x, o); }, fin);
}
// ... with the totals in FP64 for fin
template <int NV, class Fin>
__device__ __forceinline__ bool qSumDF(df (&a)[NV], const PpeBuffers& B, QCtl& c, Fin fin, bool any = true) {
    return qSumF2<NV>(a, B, c, [&](const df* t) {
        double tot[NV];
#pragma unroll
        for (int q = 0; q < NV; q++) tot[q] = dD(t[q]);
        fin(tot);
    }, any);
}

// FP64 per-thread partials summed as float-float from the warp level on (each partial split
// exactly into hi + lo to 48 bits): the per-iteration sums of the plain FP64 CG keep their
// trees off the FP64 pipe.  A tree of float-float sums over the 864k row terms rounds less
// than the sequential FP64 dot product of the reference's solver.
template <int NV, class Fin>
__device__ __forceinline__ bool qSumD(double (&v)[NV], const PpeBuffers& B, QCtl& c, Fin fin, bool any = true) {
    df a[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) a[q] = dfD(v[q]);
    return qSumDF<NV>(a, B, c, fin, any);
}

// Rows inside the persistent kernels: matrix arrays are read-only for the launch, the
// gathered vector is written by other blocks during it (plain loads, made visible by the
// barrier's fences).  forRows walks a thread's rows with the next row's length prefetched.
template <class F>
__device__ __forceinline__ void forRows(const PpeBuffers& B, int n, int t0, int T, F&& f) {
    int i = t0;
    int len = i < n ? __ldg(B.rowLen + i) : 0;
    while (i < n) {
        int in = i + T;
        int ln = in < n ? __ldg(B.rowLen + in) : 0;
        f(i, len);
        i = in;
        len = ln;
    }
}
// Balanced rows of one thread in the persistent kernels: full rounds of the grid (row =
// m T + b BS + t, T = G BS), then the remainder n - full T split evenly over the blocks, so
// every block gets the same number of rows (+-1 per thread).  A plain grid stride gives
// the first blocks one round more: at 864k rows and 152 x 1024 threads, 84 blocks did 6
// rounds and 68 did 5, and every grid sum waited for the 6-round blocks.
struct RowSet {
    int first, T, full, last;   // rows first + m T (m < full), then last (-1: none)
};
__device__ __forceinline__ RowSet rowSet(int n, int BS) {
    RowSet s;
    const int G = gridDim.x;
    s.T = G * BS;
    s.full = n / s.T;
    s.first = blockIdx.x * BS + threadIdx.x;
    const int rem = n - s.full * s.T;
    const int share = (rem + G - 1) / G;
    const int j = s.full * s.T + blockIdx.x * share + (int)threadIdx.x;
    s.last = ((int)threadIdx.x < share && j < n) ? j : -1;
    return s;
}
__device__ __forceinline__ int rowCount(const RowSet& s) { return s.full + (s.last >= 0 ? 1 : 0); }
__device__ __forceinline__ int rowAt(const RowSet& s, int m) { return m < s.full ? s.first + m * s.T : s.last; }
template <class F>
__device__ __forceinline__ void forOwn(const RowSet& s, F&& f) {
    int i = s.first;
    for (int m = 0; m < s.full; m++, i += s.T) f(i);
    if (s.last >= 0) f(s.last);
}
// The thread's rows in groups of RB: ld(i) for every row of a group (all loads in flight),
// then st(i, v) for each (a load cannot move above a store that may alias it, so a plain
// loop waits one memory latency per row)
template <int RB, class St, class LoadF, class StoreF>
__device__ __forceinline__ void forOwnGroup(const RowSet& s, LoadF&& ld, StoreF&& st) {
    const int cnt = rowCount(s);
    for (int m0 = 0; m0 < cnt; m0 += RB) {
        St v[RB];
        int ii[RB];
#pragma unroll
        for (int u = 0; u < RB; u++) {
            ii[u] = (m0 + u < cnt) ? rowAt(s, m0 + u) : -1;
            v[u] = ld(ii[u] >= 0 ? ii[u] : rowAt(s, m0));   // a valid row either way
        }
#pragma unroll
        for (int u = 0; u < RB; u++)
            if (ii[u] >= 0) st(ii[u], v[u]);
    }
}
// ELL rows with the next row's length prefetched
template <class F>
__device__ __forceinline__ void forRows(const PpeBuffers& B, const RowSet& s, F&& f) {
    const int cnt = rowCount(s);
    int i = cnt > 0 ? rowAt(s, 0) : 0;
    int len = cnt > 0 ? __ldg(B.rowLen + i) : 0;
    for (int m = 0; m < cnt; m++) {
        const int in = (m + 1 < cnt) ? rowAt(s, m + 1) : -1;
        const int ln = in >= 0 ? __ldg(B.rowLen + in) : 0;
        f(i, len);
        i = in;
        len = ln;
    }
}
__device__ __forceinline__ double qRow(const PpeBuffers& B, const double* x, int i, int len) {
    return ellRow<double, false>(B.diag, B.val, B.col, x, i, len, ellBase(B, i), B.ellStride);
}
__device__ __forceinline__ float qRowF(const PpeBuffers& B, const float* x, int i, int len) {
    return ellRow<float, false>(B.diagf, B.valf, B.col, x, i, len, ellBase(B, i), B.ellStride);
}

// Matrix-free FP32 row of the mixed solver's inner operator: the off-diagonal entries
// a_ij = coeffPPE w(r_ij; reL) are recomputed from the hi/lo position copies for the list
// entries that the assembly marked as matrix entries (mfMask), eight neighbours in flight;
// the diagonal is the assembled one.  Only the 4-byte neighbour indices are streamed.
__device__ __forceinline__ float mfWeight(float r2, float re, float invRe, int t) {
    float rinv = rsqrtf(r2);
    switch (t) {
        case 1: { float r = r2 * rinv; return re * rinv + r * invRe - 2.0f; }
        case 2: { float r = r2 * rinv; return re * rinv - r * invRe; }
        case 3: { float a = 1.0f - r2 * rinv * invRe; return a * a * a; }
        case 4: { float a = 1.0f - r2 * rinv * invRe; return a * a; }
        default: return re * rinv - 1.0f;
    }
}
__device__ __forceinline__ float mfRowF(const Dev& d, const PpeBuffers& B, const float* z, int i, float cP, float re,
                                       float invRe, int wt) {
    Mask m = B.mfMask[i];
    const float4 hi = __ldg(d.posf + i), li = __ldg(d.posLo + i);
    const int* row = d.nbr + i;
    const size_t N0 = d.N0;
    float acc[8];
#pragma unroll
    for (int u = 0; u < 8; u++) acc[u] = 0.f;
    while (m.lo | m.hi) {
        int jj[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int k = maskPop(m);
            jj[u] = (k >= 0) ? ldStream(row + (size_t)k * N0) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (jj[u] < 0) continue;
            const int j = jj[u];
            const float4 hj = __ldg(d.posf + j), lj = __ldg(d.posLo + j);
            float dx = (hj.x - hi.x) + (lj.x - li.x);
            float dy = (hj.y - hi.y) + (lj.y - li.y);
            float dz = (hj.z - hi.z) + (lj.z - li.z);
            float w = mfWeight(dx * dx + dy * dy + dz * dz, re, invRe, wt);
            acc[u] += (cP * w) * z[j];
        }
    }
    return __ldg(B.diagf + i) * z[i] + (((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7])));
}

// Compact inner operator: with s_i = 1/sqrt|A_ii| and sigma_i = sign(A_ii), the system
// A d = r is M y = c with M = diag(sigma s) A diag(s), c_i = sigma_i s_i r_i, d = s y.  M is
// symmetric (coupled rows are all equation rows, sigma = -1), has a unit diagonal and
// off-diagonals in (-1, 0): they are stored in FP16 (FP32 arithmetic), the columns as
// 16-bit offsets j - i (rows with a farther neighbour keep the 32-bit columns), 4 bytes
// per entry instead of 8, and CG on M needs no preconditioner.
__device__ __forceinline__ float h16Row(const PpeBuffers& B, const float* y, int i, int len) {
    const size_t N0 = B.ellStride, base = ellBase(B, i);
    const __half* v = B.valh + base;
    float acc[ELL_U];
#pragma unroll
    for (int u = 0; u < ELL_U; u++) acc[u] = 0.f;
    if (!__ldg(B.wideRow + i)) {
        const short* c = B.col16 + base;
        for (int k = 0; k < len; k += ELL_U) {
            if (k + ELL_U < len) {
#pragma unroll
                for (int u = 0; u < ELL_U; u += 2) {
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(c + (size_t)(k + ELL_U + u) * N0));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(v + (size_t)(k + ELL_U + u) * N0));
                }
            }
            int cc[ELL_U];
            float vv[ELL_U];
#pragma unroll
            for (int u = 0; u < ELL_U; u++) {
                bool ok = k + u < len;
                cc[u] = ok ? i + (int)__ldg(c + (size_t)(k + u) * N0) : i;
                vv[u] = ok ? __half2float(__ldg(v + (size_t)(k + u) * N0)) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < ELL_U; u++) acc[u] += vv[u] * y[cc[u]];
        }
    } else {
        const int* c = B.col + base;
        for (int k = 0; k < len; k += ELL_U) {
            int cc[ELL_U];
            float vv[ELL_U];
#pragma unroll
            for (int u = 0; u < ELL_U; u++) {
                bool ok = k + u < len;
                cc[u] = ok ? ldStream(c + (size_t)(k + u) * N0) : i;
                vv[u] = ok ? __half2float(__ldg(v + (size_t)(k + u) * N0)) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < ELL_U; u++) acc[u] += vv[u] * y[cc[u]];
        }
    }
    return y[i] + (((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7])));
}

// ------------------------------------------------------------------ staged ELL tiles
// The FP32 inner SpMV with the matrix streamed through shared memory: a block owns the
// 256-row tiles t = blockIdx.x + m gridDim.x (the rows its threads own in every other
// phase); each tile's column and value slices (1 KB each, column-major ELL) are copied by
// the bulk-copy engine (cp.async.bulk, completion counted on an mbarrier) in chunks of
// TS_CH slices into a TS_NS-stage ring, up to TS_NS - 1 chunks ahead of the threads, which
// read their row's entries from shared memory and gather z.  The engine keeps the HBM
// stream in flight independently of the threads' gather latencies.  Every mbarrier wait
// is bounded; a wait that runs out sets the abort word (mps_grid.cuh) and the block stops
// consuming, drains the copies it issued (again bounded) and returns at the next barrier.
#define TS_CH 8
#define TS_NS 3
#define TS_SPIN (1 << 20)
struct TsStage {
    int col[TS_CH][QB];
    float val[TS_CH][QB];
};
#define TS_MAXT 128   // tiles per block held in shared memory
struct TsSmem {
    TsStage st[TS_NS];
    unsigned long long full[TS_NS], empty[TS_NS];
    int tlen[TS_MAXT];
};
// bounded wait; false when it ran out
__device__ __forceinline__ bool mbarWait(unsigned long long* b, unsigned parity) { return mbarWaitN(b, parity, TS_SPIN); }
// Chunk walk of a block: its tiles in order (m-th tile = blockIdx.x + m gridDim.x, length
// tlen[m] = longest row), ceil(len / TS_CH) chunks each.
struct TsWalk {
    int m, chunk;
};
__device__ __forceinline__ bool tsNext(const TsSmem& sm, int mt, TsWalk& w) {
    while (w.m < mt) {
        if (w.chunk * TS_CH < sm.tlen[w.m]) return true;
        w.m++;
        w.chunk = 0;
    }
    return false;
}
// issue one chunk (thread 0): slices [c TS_CH, min(L, (c+1) TS_CH)) of the walk's tile
__device__ __forceinline__ void tsIssue(TsSmem& sm, const PpeBuffers& B, const TsWalk& w, unsigned q, bool& ok) {
    const int s = q % TS_NS;
    const unsigned use = q / TS_NS;
    if (use > 0 && !mbarWait(&sm.empty[s], (use - 1) & 1)) { ok = false; return; }
    const int L = sm.tlen[w.m];
    const int k0 = w.chunk * TS_CH, nsl = min(TS_CH, L - k0);
    const size_t r0 = (size_t)(blockIdx.x + w.m * gridDim.x) * QB;
    mbarExpectTx(&sm.full[s], (unsigned)(nsl * QB * (sizeof(int) + sizeof(float))));
    for (int u = 0; u < nsl; u++) {   // a tile's QB rows lie in one slice (the slice height is a multiple of QB)
        size_t e = ellBase(B, (int)r0) + (size_t)(k0 + u) * B.ellStride;
        bulkG2S(sm.st[s].col[u], B.col + e, QB * sizeof(int), &sm.full[s]);
        bulkG2S(sm.st[s].val[u], B.valf + e, QB * sizeof(float), &sm.full[s]);
    }
}

// One staged SpMV pass over the block's tiles: y_i = A_ii z_i + sum_k valf z[col] for the
// thread's row of every tile, then rowDone(i, y_i) (rows below the live count only).
// gq counts the chunks consumed, the same in every thread; returns false when a wait ran
// out (the abort word is then set; the copies issued are drained, bounded, before return).
template <class F>
__device__ __forceinline__ bool tsSpmv(TsSmem& sm, const PpeBuffers& B, const float* z, int n, int mt, unsigned& gq,
                                       F&& rowDone) {
    bool ok = true;
    TsWalk prod = {0, 0};
    unsigned qp = gq, q = gq;
    if (threadIdx.x == 0)
        for (int k = 0; k < TS_NS - 1 && ok && tsNext(sm, mt, prod); k++) { tsIssue(sm, B, prod, qp, ok); qp++; prod.chunk++; }
    for (int m = 0; m < mt; m++) {
        const int row = (blockIdx.x + m * gridDim.x) * QB + threadIdx.x;
        const int len = (row < n) ? __ldg(B.rowLen + row) : 0;
        const int L = sm.tlen[m];
        float acc[TS_CH];
#pragma unroll
        for (int u = 0; u < TS_CH; u++) acc[u] = 0.f;
        for (int c = 0; c * TS_CH < L; c++) {
            if (threadIdx.x == 0 && ok && tsNext(sm, mt, prod)) { tsIssue(sm, B, prod, qp, ok); qp++; prod.chunk++; }
            const int st = q % TS_NS;
            bool got = ok && mbarWait(&sm.full[st], (q / TS_NS) & 1);
            got = __all_sync(0xffffffffu, got);
            if (got) {
                const int k0 = c * TS_CH;
#pragma unroll
                for (int u = 0; u < TS_CH; u++)
                    if (k0 + u < len) acc[u] += sm.st[st].val[u][threadIdx.x] * z[sm.st[st].col[u][threadIdx.x]];
            } else {
                ok = false;
            }
            __syncwarp();
            if ((threadIdx.x & 31) == 0) mbarArrive(&sm.empty[st]);
            q++;
        }
        if (row < n)
            rowDone(row, __ldg(B.diagf + row) * z[row] +
                             (((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]))));
    }
    // a wait that ran out: stop, and let the copies this block issued land before leaving
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
            atomicExch(B.bar + QB_ABT, 1u);
            for (unsigned k = q; k < qp; k++) mbarWait(&sm.full[k % TS_NS], (k / TS_NS) & 1);
        }
        __syncthreads();
        return false;
    }
    gq = q;
    return true;
}

// Mixed solver: FP64 residual r = b - A x and its norm, FP32 inner CG on r / ||r|| to
// the relative tolerance eta_k, x += ||r|| d in FP64, repeated until ||r|| < tol ||b||.
// eta_k = max(eta, tol ||b|| / (2 ||r_k||)): an inner solve stops once its correction
// brings the outer residual to half the tolerance, so the last one does not over-solve;
// eta = 1e-6 is near the FP32 recurrence's attainable accuracy.
// Inner operator of k_mx_solve: the assembled FP32 ELL matrix with Jacobi preconditioning,
// the matrix-free FP32 operator with Jacobi preconditioning, or the compact scaled operator.
enum { OP_ELL32 = 0, OP_MATFREE = 1, OP_H16 = 2, OP_TILED = 3 };
template <int OP>
__global__ void __launch_bounds__(OP == 3 ? QB : QBX, OP == 3 ? 4 : 1) k_mx_solve(Dev d, PpeBuffers B, double tol, int maxIter, double eta2) {
    __shared__ QLocal qL;   // this block's copy of the solver scalars and flags
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    extern __shared__ __align__(128) unsigned char dynSmem[];
    const int n = liveN(d);
    const float cP = (float)d.P.coeffPPE, re = (float)d.P.reL, invRe = (float)(1.0 / d.P.reL);
    const int wt = d.P.weightType;
    // grid-stride rounds (at any moment the blocks work on one contiguous window of rows,
    // so the column slices of the ELL arrays stream through DRAM pages in order), the
    // remainder split evenly over the blocks
    constexpr int BS = (OP == OP_TILED) ? QB : QBX;
    const RowSet rs = rowSet(n, BS);   // this thread's rows
    QCtl c = {0u};
    // staged tiles: the block's tile lengths and the mbarriers of the ring
    TsSmem& sm = *reinterpret_cast<TsSmem*>(dynSmem);
    const int ntiles = (n + QB - 1) / QB;
    const int mt = (ntiles > (int)blockIdx.x) ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    unsigned gq = 0u;   // chunks consumed so far (the same count in every thread of the block)
    if (OP == OP_TILED) {
        if (threadIdx.x == 0) {
            for (int st = 0; st < TS_NS; st++) {
                mbarInit(&sm.full[st], 1u);
                mbarInit(&sm.empty[st], QB / 32);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int m = threadIdx.x; m < TS_MAXT; m += QB) sm.tlen[m] = 0;
        __syncthreads();
        for (int m = 0; m < mt; m++) {
            const int row = (blockIdx.x + m * gridDim.x) * QB + threadIdx.x;
            int len = (row < n) ? __ldg(B.rowLen + row) : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
            if ((threadIdx.x & 31) == 0) atomicMax(&sm.tlen[m], len);
        }
        __syncthreads();
    }
    if (OP == OP_H16) {
        // scaling, then the compact copy of the FP32 matrix
        forOwn(rs, [&](int i) {
            double dd = __ldg(B.diag + i);
            double sc = 1.0 / sqrt(fabs(dd));
            B.sclf[i] = (float)sc;
            B.sgs[i] = (float)(dd < 0.0 ? -sc : sc);
        });
        if (!qBarrier(B, c)) return;
        forRows(B, rs, [&](int i, int len) {
            const float si = B.sgs[i];
            unsigned char wide = 0;
            const size_t base = ellBase(B, i);
            for (int k = 0; k < len; k++) {
                size_t e = base + (size_t)k * B.ellStride;
                int j = __ldg(B.col + e);
                B.valh[e] = __float2half_rn(si * __ldg(B.valf + e) * B.sclf[j]);
                int off = j - i;
                if (off < -32768 || off > 32767) wide = 1;
                B.col16[e] = (short)off;
            }
            B.wideRow[i] = wide;
        });
        if (!qBarrier(B, c)) return;
    }
    {
        double v[2] = {0.0, 0.0};
        forRows(B, rs, [&](int i, int len) {
            double r = B.b[i] - qRow(B, B.x, i, len);
            B.r[i] = r;
            v[0] += r * r;
            v[1] += B.b[i] * B.b[i];
        });
        if (!qSum<2>(v, B, c, [&](const double* t) {
                qS[S_RR] = t[0];
                qS[S_BB] = t[1];
                double thr = tol * tol * t[1];
                if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
                qS[S_THR] = thr;
                qS[S_SCALE] = sqrt(t[0] / (t[1] > 0 ? t[1] : 1.0));
                qS[S_SQRT] = sqrt(t[0]);
                qS[S_INV] = 1.0 / sqrt(t[0]);
                qS[S_ETA2] = fmax(eta2, 0.25 * thr / t[0]);
                qF[0] = (t[1] == 0.0 || t[0] < thr) ? 1 : 0;
                qF[1] = 0;
                qF[3] = 0;
                if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
            }))
            return;
    }
    int total = 0, refine = 0;
    while (!vi(qF) && total < maxIter && refine <= 20) {
        // inner start: rf = r / ||r|| (compact operator: sigma s r / ||r||), z = M^-1 rf, x_f = 0
        {
            const double inv = vd(qS + S_INV);
            df a[2] = {dfF(0.f), dfF(0.f)};
            forOwn(rs, [&](int i) {
                float r = (float)(B.r[i] * inv);
                if (OP == OP_H16) r *= B.sgs[i];
                float z = (OP == OP_H16) ? r : r * __ldg(B.diagInvf + i);
                B.rf[i] = r; B.zf[i] = z; B.xf[i] = 0.f;
                a[0] += prod2(r, z);
                a[1] += prod2(r, r);
            });
            if (!qSumDF<2>(a, B, c, [&](const double* t) { qS[S_RZ] = t[0]; qS[S_RR0] = t[1]; qF[3] = 0; }))
                return;
        }
        int inner = 0;
        while (true) {
            {
                const float beta = inner ? (float)vd(qS + S_BETA) : 0.f;
                df a[1] = {dfF(0.f)};
                if (OP == OP_TILED) {
                    bool okp = tsSpmv(sm, B, B.zf, n, mt, gq, [&](int i, float q) {
                        float z = B.zf[i];
                        float ap = inner ? q + beta * B.Apf[i] : q;
                        float p = inner ? z + beta * B.pf[i] : z;
                        B.Apf[i] = ap; B.pf[i] = p;
                        a[0] += prod2(p, ap);
                    });
                    (void)okp;   // an ran-out wait sets the abort word: the reduction below returns false
                } else forRows(B, rs, [&](int i, int len) {
                    float q = (OP == OP_MATFREE) ? mfRowF(d, B, B.zf, i, cP, re, invRe, wt)
                            : (OP == OP_H16)   ? h16Row(B, B.zf, i, len)
                                               : qRowF(B, B.zf, i, len);
                    float z = B.zf[i];
                    float ap = inner ? q + beta * B.Apf[i] : q;
                    float p = inner ? z + beta * B.pf[i] : z;
                    B.Apf[i] = ap; B.pf[i] = p;
                    a[0] += prod2(p, ap);
                });
                if (!qSumDF<1>(a, B, c, [&](const double* t) { qS[S_PAP] = t[0]; qS[S_ALPHA] = qS[S_RZ] / t[0]; }))
                    return;
            }
            {
                const float alpha = (float)vd(qS + S_ALPHA);
                df a[2] = {dfF(0.f), dfF(0.f)};
                struct VR { float x, p, r, q, m; };
                forOwnGroup<3, VR>(rs, [&](int i) {
                    VR v;
                    v.x = B.xf[i]; v.p = B.pf[i]; v.r = B.rf[i]; v.q = B.Apf[i];
                    v.m = (OP == OP_H16) ? 1.f : __ldg(B.diagInvf + i);
                    return v;
                }, [&](int i, const VR& v) {
                    const float r = v.r - alpha * v.q;
                    const float z = (OP == OP_H16) ? r : r * v.m;
                    B.xf[i] = v.x + alpha * v.p; B.rf[i] = r; B.zf[i] = z;
                    a[0] += prod2(r, z);
                    a[1] += prod2(r, r);
                });
                if (!qSumDF<2>(a, B, c, [&](const double* t) {
                        qF[1] += 1;
                        qS[S_BETA] = t[0] / qS[S_RZ];
                        qS[S_RZ] = t[0];
                        if (t[1] < qS[S_ETA2] * qS[S_RR0] || !(t[1] == t[1])) qF[3] = 1;
                    }))
                    return;
            }
            inner++;
            if (vi(qF + 3) || total + inner >= maxIter || inner >= 400) break;
        }
        total += inner;
        {
            const double sc = vd(qS + S_SQRT);
            forOwn(rs, [&](int i) {
                B.x[i] += sc * (double)((OP == OP_H16) ? B.xf[i] * B.sclf[i] : B.xf[i]);
            });
            if (!qBarrier(B, c)) return;
        }
        {
            double v[1] = {0.0};
            forRows(B, rs, [&](int i, int len) {
                double r = B.b[i] - qRow(B, B.x, i, len);
                B.r[i] = r;
                v[0] += r * r;
            });
            if (!qSum<1>(v, B, c, [&](const double* t) {
                    qS[S_RR] = t[0];
                    qS[S_SQRT] = sqrt(t[0]);
                    qS[S_INV] = 1.0 / sqrt(t[0]);
                    qS[S_ETA2] = fmax(eta2, 0.25 * qS[S_THR] / t[0]);
                    if (t[0] < qS[S_THR]) qF[0] = 1;
                    if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
                    qF[4] += 1;
                }))
                return;
        }
        refine++;
    }
    qStore(B, qL);
}

// ------------------------------------------------------------------ shared-memory vectors
// The mixed solver with the FP32 inner-CG vectors of each block's rows (Ap, p, r, x: 16
// bytes per row, fewer of them above 1.7M rows) in shared memory from the first inner iteration
// to the last; only z, the
// vector every block gathers through the matrix columns, goes through global memory.  A
// block's rows are those of the grid-stride rounds (RowSet: at any moment all blocks
// stream adjacent slices of the column-major ELL arrays, which measured 28% faster than one
// contiguous range per block), and the m-th row of thread t sits at slot m BS + t of the
// block's vectors.  The vector pass of an iteration is then shared-memory work plus one
// coalesced store of z.

// The thread's rows of a RowSet with their shared-memory slot l = m BS + t (m-th row of the
// thread), f(l, i, len) with the next row's length prefetched; forOwnL without the length.
template <class F>
__device__ __forceinline__ void forRowsL(const PpeBuffers& B, const RowSet& s, F&& f) {
    const int cnt = rowCount(s);
    int i = cnt > 0 ? rowAt(s, 0) : 0;
    int len = cnt > 0 ? __ldg(B.rowLen + i) : 0;
    for (int m = 0; m < cnt; m++) {
        const int in = (m + 1 < cnt) ? rowAt(s, m + 1) : -1;
        const int ln = in >= 0 ? __ldg(B.rowLen + in) : 0;
        f(m * (int)blockDim.x + (int)threadIdx.x, i, len);
        i = in;
        len = ln;
    }
}
template <class F>
__device__ __forceinline__ void forOwnL(const RowSet& s, F&& f) {
    const int cnt = rowCount(s);
    for (int m = 0; m < cnt; m++) f(m * (int)blockDim.x + (int)threadIdx.x, rowAt(s, m));
}

// Scalars of a mixed solve from the sums r.r, b.b (LEARNED: also r.q and q.q) of its start.
template <bool LEARNED>
__device__ __forceinline__ void mxStart(QLocal& qL, const double* t, double tol, double eta2) {
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    double th = 0.0, rr = t[0];
    if (LEARNED) {
        // a non-finite correction keeps the start x (theta = 0, its residual as is)
        const double rq = t[LEARNED ? 2 : 0], qq = t[LEARNED ? 3 : 0];
        if (qq > 0.0 && qq < 1.0 / 0.0 && rq == rq && fabs(rq) < 1.0 / 0.0) {
            th = rq / qq;
            rr = fmax(t[0] - th * rq, 0.0);
        }
    }
    qS[S_OMEGA] = th;
    qS[S_RR] = rr;
    qS[S_BB] = t[1];
    double thr = tol * tol * t[1];
    if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
    qS[S_THR] = thr;
    qS[S_SCALE] = sqrt(rr / (t[1] > 0 ? t[1] : 1.0));
    qS[S_SQRT] = sqrt(rr);
    qS[S_INV] = 1.0 / sqrt(rr);
    qS[S_ETA2] = fmax(eta2, 0.25 * thr / rr);
    qF[0] = (t[1] == 0.0 || rr < thr) ? 1 : 0;
    qF[1] = 0;
    qF[3] = 0;
    if (!(rr == rr)) { qF[0] = 1; qF[2] = 1; }
}
// Set-up of the shared-memory mixed solve: FP64 residual of the warm start, ||r||^2 and
// ||b||^2 and the solver scalars; with a learned correction c (B.cdir, with q = A c in
// B.cq) the residual r_e of the start x_e is already in B.r (the learned start's features
// read it), and the pass forms the dot products r.q and q.q, the residual-minimising step
// theta = r.q / q.q (the start x + theta c is never worse than x in the residual norm; its
// residual norm follows algebraically) and the update of x and r.  Returns false when a
// barrier wait ran out.
template <bool LEARNED>
__device__ __forceinline__ bool mxSetup(const PpeBuffers& B, const RowSet& rs, QCtl& c, QLocal& qL, double tol,
                                        double eta2) {
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    double v[LEARNED ? 4 : 2] = {};
    if (LEARNED) {
        forOwn(rs, [&](int i) {
            const double bi = B.b[i], r = B.r[i];
            const double q = (double)__ldg(B.cq + i);
            v[0] += r * r;
            v[1] += bi * bi;
            v[LEARNED ? 2 : 0] += r * q;
            v[LEARNED ? 3 : 0] += q * q;
        });
    } else {
        forRows(B, rs, [&](int i, int len) {
            const double bi = B.b[i];
            const double r = bi - qRow(B, B.x, i, len);
            B.r[i] = r;
            v[0] += r * r;
            v[1] += bi * bi;
        });
    }
    if (!qSum<LEARNED ? 4 : 2>(v, B, c, [&](const double* t) { mxStart<LEARNED>(qL, t, tol, eta2); }))
        return false;
    if (LEARNED && vd(qS + S_OMEGA) != 0.0) {   // x += theta c, r -= theta q on the thread's own rows
        const double th = vd(qS + S_OMEGA);
        forOwn(rs, [&](int i) {
            B.x[i] += th * (double)__ldg(B.cdir + i);
            B.r[i] -= th * (double)__ldg(B.cq + i);
        });
    }
    return true;
}

// NV of the four inner vectors are in shared memory: Ap, p, r, x in this order (the ones an
// iteration touches most first), the others in B.rf and B.xf.  The FP32 step scalars
// are the bits of the FP64 quotients of the sums, without an FP64 division on one thread between
// two grid sums (108k learned start 4.76 ms with them, 4.63 without; 864k steps 19.17 / 18.94).
template <bool LEARNED, int NV>
__global__ void __launch_bounds__(QBX, 1) k_mx_own(Dev d, PpeBuffers B, double tol, int maxIter, double eta2, int cap) {
    __shared__ QLocal qL;   // this block's copy of the solver scalars and flags
    __shared__ df rz, stop2;   // inner solve: r.z, and the squared residual norm that ends it
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    extern __shared__ __align__(128) unsigned char dynSmem[];
    float* const sap = reinterpret_cast<float*>(dynSmem);   // A p
    float* const sp = sap + cap;                             // search direction
    float* const sr = sp + cap;                              // inner residual
    float* const sx = sr + cap;                              // inner correction x_f
    auto R = [&](int l, int i) -> float& { return NV >= 3 ? sr[l] : B.rf[i]; };
    auto X = [&](int l, int i) -> float& { return NV >= 4 ? sx[l] : B.xf[i]; };
    const int n = liveN(d);
    const RowSet rs = rowSet(n, QBX);   // this thread's rows (rowCount(rs) * QBX <= cap)
    QCtl c = {0u};
    if (!mxSetup<LEARNED>(B, rs, c, qL, tol, eta2)) return;
    int total = 0, refine = 0;
    while (!vi(qF) && total < maxIter && refine <= 20) {
        {   // inner start: r_f = r / ||r||, z = M^-1 r_f, x_f = 0
            const double inv = vd(qS + S_INV);
            df a[2] = {dfF(0.f), dfF(0.f)};
            forOwnL(rs, [&](int l, int i) {
                const float r = (float)(B.r[i] * inv);
                const float z = r * __ldg(B.diagInvf + i);
                R(l, i) = r; X(l, i) = 0.f;
                B.zf[i] = z;
                a[0] += prod2(r, z);
                a[1] += prod2(r, r);
            });
            if (!qSumF2<2>(a, B, c, [&](const df* t) {
                    rz = t[0];
                    stop2 = dfD(dD(t[1]) * qS[S_ETA2]);
                    qF[3] = 0;
                }))
                return;
        }
        int inner = 0;
        while (true) {
            {   // Ap = A z + beta Ap, p = z + beta p, p.Ap
                const float beta = inner ? vf(qL.scalf + SF_BETA) : 0.f;
                df a[1] = {dfF(0.f)};
                forRowsL(B, rs, [&](int l, int i, int len) {
                    const float q = qRowF(B, B.zf, i, len);
                    const float z = B.zf[i];
                    const float ap = inner ? q + beta * sap[l] : q;
                    const float p = inner ? z + beta * sp[l] : z;
                    sap[l] = ap; sp[l] = p;
                    a[0] += prod2(p, ap);
                });
                if (!qSumF2<1>(a, B, c, [&](const df* t) { qL.scalf[SF_ALPHA] = divF(rz, t[0]); })) return;
            }
            {   // x_f += alpha p, r -= alpha Ap, z = M^-1 r; r.z, r.r
                const float alpha = vf(qL.scalf + SF_ALPHA);
                df a[2] = {dfF(0.f), dfF(0.f)};
                const int cnt = rowCount(rs);
                for (int m0 = 0; m0 < cnt; m0 += 4) {
                    float mi[4], ro[4], xo[4];
                    int ii[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        ii[u] = (m0 + u < cnt) ? rowAt(rs, m0 + u) : -1;
                        mi[u] = (ii[u] >= 0) ? __ldg(B.diagInvf + ii[u]) : 0.f;
                        if (NV < 3) ro[u] = (ii[u] >= 0) ? B.rf[ii[u]] : 0.f;
                        if (NV < 4) xo[u] = (ii[u] >= 0) ? B.xf[ii[u]] : 0.f;
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (ii[u] < 0) continue;
                        const int l = (m0 + u) * (int)blockDim.x + (int)threadIdx.x;
                        const float r = (NV < 3 ? ro[u] : sr[l]) - alpha * sap[l];
                        const float z = r * mi[u];
                        X(l, ii[u]) = (NV < 4 ? xo[u] : sx[l]) + alpha * sp[l];
                        R(l, ii[u]) = r;
                        B.zf[ii[u]] = z;
                        a[0] += prod2(r, z);
                        a[1] += prod2(r, r);
                    }
                }
                if (!qSumF2<2>(a, B, c, [&](const df* t) {
                        qF[1] += 1;
                        qL.scalf[SF_BETA] = divF(t[0], rz);
                        rz = t[0];
                        if (t[1] < stop2 || !(t[1].h == t[1].h)) qF[3] = 1;
                    }))
                    return;
            }
            inner++;
            if (vi(qF + 3) || total + inner >= maxIter || inner >= 400) break;
        }
        total += inner;
        {   // x += ||r|| x_f (FP64)
            const double sc = vd(qS + S_SQRT);
            forOwnL(rs, [&](int l, int i) { B.x[i] += sc * (double)X(l, i); });
            if (!qBarrier(B, c)) return;
        }
        {   // FP64 residual r = b - A x
            double v[1] = {0.0};
            forRows(B, rs, [&](int i, int len) {
                const double r = B.b[i] - qRow(B, B.x, i, len);
                B.r[i] = r;
                v[0] += r * r;
            });
            if (!qSum<1>(v, B, c, [&](const double* t) {
                    qS[S_RR] = t[0];
                    qS[S_SQRT] = sqrt(t[0]);
                    qS[S_INV] = 1.0 / sqrt(t[0]);
                    qS[S_ETA2] = fmax(eta2, 0.25 * qS[S_THR] / t[0]);
                    if (t[0] < qS[S_THR]) qF[0] = 1;
                    if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
                    qF[4] += 1;
                }))
                return;
        }
        refine++;
    }
    qStore(B, qL);
}
// Kernel and shared memory of the mixed solve with nv vectors there
static const void* ownKernel(bool learned, int nv) {
    if (learned) return nv >= 4 ? (const void*)k_mx_own<true, 4> : nv == 3 ? (const void*)k_mx_own<true, 3> : (const void*)k_mx_own<true, 2>;
    return nv >= 4 ? (const void*)k_mx_own<false, 4> : nv == 3 ? (const void*)k_mx_own<false, 3> : (const void*)k_mx_own<false, 2>;
}

// FP64 residual row of the refinement without a pass in between: x_j + d_j is formed from
// the FP64 iterate and the FP32 correction of the inner solve as the owner of j forms it.
__device__ __forceinline__ double qRowPlus(const PpeBuffers& B, const double* x, const float* dx, int i, int len) {
    double acc[ELL_U];
#pragma unroll
    for (int u = 0; u < ELL_U; u++) acc[u] = 0.0;
    const size_t base = ellBase(B, i), N0 = B.ellStride;
    const double* v = B.val + base;
    const int* c = B.col + base;
    for (int k = 0; k < len; k += ELL_U) {
        int cc[ELL_U];
        double vv[ELL_U];
#pragma unroll
        for (int u = 0; u < ELL_U; u++) {
            bool ok = k + u < len;
            cc[u] = ok ? ldStream(c + (size_t)(k + u) * N0) : i;
            vv[u] = ok ? ldStream(v + (size_t)(k + u) * N0) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < ELL_U; u++) acc[u] += vv[u] * (x[cc[u]] + (double)dx[cc[u]]);
    }
    return __ldg(B.diag + i) * (x[i] + (double)dx[i]) +
           (((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7])));
}

// Mixed solver with the pipelined inner CG (Ghysels & Vanroose, "Hiding global
// synchronization latency in the preconditioned Conjugate Gradient algorithm", Parallel
// Computing 40, 2014, Alg. 3), Jacobi M = diag^-1 applied on the fly: with u = M r,
// q = M s and m = M w recomputed from r, s and w, the recurrences kept are
//   z = A m + beta z,  s = w + beta s,  p = M r + beta p,  x += alpha p,
//   r -= alpha s,      w -= alpha z,    m' = M w
// and the three dot products (r.u, w.u, r.r) of the next iteration are summed in the same
// pass: one grid barrier per inner iteration (the standard form needs two).  m is double
// buffered (its owner writes m' while neighbours gather m).  The FP64 refinement forms
// r = b - A (x + d) in the pass that stores x + d into the other FP64 buffer, and starts
// the next inner solve there (u0 = M r), so a refinement costs two barriers.
__global__ void __launch_bounds__(QBX, 1) k_mx_pipe(Dev d, PpeBuffers B, double tol, int maxIter, double eta2) {
    __shared__ QLocal qL;   // this block's copy of the solver scalars and flags
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    const int n = liveN(d);
    const RowSet rs = rowSet(n, QBX);   // this thread's rows
    QCtl c = {0u};
    double* xa = B.x;      // current FP64 iterate
    double* xb = B.xalt;   // the next one
    float* mA = B.zf;      // u0, then m of odd iterations
    float* mB = B.mf2;     // m of even iterations
    {
        double v[2] = {0.0, 0.0};
        forRows(B, rs, [&](int i, int len) {
            double r = B.b[i] - qRow(B, xa, i, len);
            B.r[i] = r;
            float rf = (float)r;
            B.rf[i] = rf;
            mA[i] = rf * __ldg(B.diagInvf + i);
            v[0] += r * r;
            v[1] += B.b[i] * B.b[i];
        });
        if (!qSum<2>(v, B, c, [&](const double* t) {
                qS[S_RR] = t[0];
                qS[S_BB] = t[1];
                double thr = tol * tol * t[1];
                if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
                qS[S_THR] = thr;
                qS[S_SCALE] = sqrt(t[0] / (t[1] > 0 ? t[1] : 1.0));
                qS[S_ETA2] = fmax(eta2, 0.25 * thr / t[0]);
                qF[0] = (t[1] == 0.0 || t[0] < thr) ? 1 : 0;
                qF[1] = 0;
                if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
            }))
            return;
    }
    int total = 0, refine = 0;
    while (!vi(qF) && total < maxIter && refine <= 20) {
        // inner start: w0 = A u0, m0 = M w0; gamma0 = r.u, delta0 = w.u, rho0 = r.r
        {
            df a[3] = {dfF(0.f), dfF(0.f), dfF(0.f)};
            forRows(B, rs, [&](int i, int len) {
                const float w = qRowF(B, mA, i, len);
                const float u = mA[i], r = B.rf[i];
                B.wf[i] = w;
                mB[i] = w * __ldg(B.diagInvf + i);
                a[0] += prod2(r, u);
                a[1] += prod2(w, u);
                a[2] += prod2(r, r);
            });
            if (!qSumDF<3>(a, B, c, [&](const double* t) {
                    qF[3] = 0;
                    qS[S_RZ] = t[0];
                    qS[S_RR0] = t[2];
                    qS[S_BETA] = 0.0;
                    // the PPE matrix and its Jacobi preconditioner are negative definite:
                    // r.u and w.u share their sign and alpha > 0
                    const double al = t[0] / t[1];
                    if (al > 0.0 && al < 1e300) qS[S_ALPHA] = al;
                    else qF[3] = 1;   // zero residual or breakdown: nothing to solve
                }))
                return;
        }
        int inner = 0;
        while (!vi(qF + 3) && total + inner < maxIter && inner < 400) {
            const float alpha = (float)vd(qS + S_ALPHA), beta = (float)vd(qS + S_BETA);
            const float* mc = (inner & 1) ? mA : mB;
            float* mn = (inner & 1) ? mB : mA;
            const bool first = inner == 0;
            df a[3] = {dfF(0.f), dfF(0.f), dfF(0.f)};
            forRows(B, rs, [&](int i, int len) {
                const float an = qRowF(B, mc, i, len);   // A m
                const float di = __ldg(B.diagInvf + i);
                float w = B.wf[i], r = B.rf[i];
                float z = first ? an : an + beta * B.qzf[i];
                float sv = first ? w : w + beta * B.Apf[i];
                float p = first ? r * di : r * di + beta * B.pf[i];
                float x = first ? alpha * p : B.xf[i] + alpha * p;
                r -= alpha * sv;
                w -= alpha * z;
                B.qzf[i] = z; B.Apf[i] = sv; B.pf[i] = p; B.xf[i] = x;
                B.rf[i] = r; B.wf[i] = w;
                const float u = r * di;
                mn[i] = w * di;
                a[0] += prod2(r, u);
                a[1] += prod2(w, u);
                a[2] += prod2(r, r);
            });
            if (!qSumDF<3>(a, B, c, [&](const double* t) {
                    qF[1] += 1;
                    if (t[2] < qS[S_ETA2] * qS[S_RR0] || !(t[2] == t[2])) { qF[3] = 1; return; }
                    const double g0 = qS[S_RZ], al = qS[S_ALPHA];
                    const double bt = t[0] / g0;
                    const double aln = t[0] / (t[1] - bt * t[0] / al);
                    if (!(aln > 0.0 && aln < 1e300 && bt >= 0.0)) { qF[3] = 1; return; }
                    qS[S_BETA] = bt;
                    qS[S_ALPHA] = aln;
                    qS[S_RZ] = t[0];
                }))
                return;
            inner++;
        }
        total += inner;
        // refinement: x' = x + d into the other buffer, r = b - A x', next inner start u0
        {
            const bool any = inner > 0;
            double v[1] = {0.0};
            forRows(B, rs, [&](int i, int len) {
                double r;
                if (any) {
                    xb[i] = xa[i] + (double)B.xf[i];
                    r = B.b[i] - qRowPlus(B, xa, B.xf, i, len);
                } else {
                    xb[i] = xa[i];
                    r = B.r[i];
                }
                B.r[i] = r;
                float rf = (float)r;
                B.rf[i] = rf;
                mA[i] = rf * __ldg(B.diagInvf + i);
                v[0] += r * r;
            });
            if (!qSum<1>(v, B, c, [&](const double* t) {
                    qS[S_RR] = t[0];
                    qS[S_ETA2] = fmax(eta2, 0.25 * qS[S_THR] / t[0]);
                    if (t[0] < qS[S_THR]) qF[0] = 1;
                    if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
                    qF[4] += 1;
                }))
                return;
            double* tx = xa; xa = xb; xb = tx;
        }
        refine++;
    }
    if (xa != B.x)
        forOwn(rs, [&](int i) { B.x[i] = xa[i]; });
    qStore(B, qL);
}

// Plain FP64 Jacobi-PCG (Eigen's ConjugateGradient with its diagonal preconditioner,
// src/MpsPressure.cpp:424-445): z = invdiag * r, stop when ||r||^2 < tol^2 ||b||^2.
__global__ void __launch_bounds__(QBC, 1) k_cg_solve(Dev d, PpeBuffers B, double tol, int maxIter) {
    __shared__ QLocal qL;   // this block's copy of the solver scalars and flags
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    const int n = liveN(d);
    // grid-stride rounds (at any moment the blocks work on one contiguous window of rows,
    // so the column slices of the ELL arrays stream through DRAM pages in order), the
    // remainder split evenly over the blocks
    const RowSet rs = rowSet(n, QBC);   // this thread's rows
    QCtl c = {0u};
    {
        double v[3] = {0.0, 0.0, 0.0};
        forRows(B, rs, [&](int i, int len) {
            double di = 1.0 / __ldg(B.diag + i);
            double r = B.b[i] - qRow(B, B.x, i, len);
            double z = r * di;
            B.dinv[i] = di; B.r[i] = r; B.z[i] = z;
            v[0] += r * z; v[1] += r * r; v[2] += B.b[i] * B.b[i];
        });
        if (!qSum<3>(v, B, c, [&](const double* t) {
                qS[S_RZ] = t[0]; qS[S_RR] = t[1]; qS[S_BB] = t[2];
                double thr = tol * tol * t[2];
                if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
                qS[S_THR] = thr;
                qS[S_SCALE] = sqrt(t[1] / (t[2] > 0 ? t[2] : 1.0));
                qF[0] = (t[2] == 0.0 || t[1] < thr) ? 1 : 0;
                qF[1] = 0;
                if (!(t[0] == t[0]) || !(t[1] == t[1])) { qF[0] = 1; qF[2] = 1; }
            }))
            return;
    }
    int it = 0;
    while (!vi(qF) && it < maxIter) {
        {
            const double beta = it ? vd(qS + S_BETA) : 0.0;
            double v[1] = {0.0};
            forRows(B, rs, [&](int i, int len) {
                double q = qRow(B, B.z, i, len);
                double z = B.z[i];
                double ap = it ? q + beta * B.Ap[i] : q;
                double p = it ? z + beta * B.p[i] : z;
                B.Ap[i] = ap; B.p[i] = p;
                v[0] += p * ap;
            });
            if (!qSum<1>(v, B, c, [&](const double* t) { qS[S_PAP] = t[0]; qS[S_ALPHA] = qS[S_RZ] / t[0]; }))
                return;
        }
        {
            const double alpha = vd(qS + S_ALPHA);
            double v[2] = {0.0, 0.0};
            struct VR { double x, p, r, q, m; };
            forOwnGroup<4, VR>(rs, [&](int i) {
                VR w;
                w.x = B.x[i]; w.p = B.p[i]; w.r = B.r[i]; w.q = B.Ap[i]; w.m = B.dinv[i];
                return w;
            }, [&](int i, const VR& w) {
                const double r = w.r - alpha * w.q;
                const double z = r * w.m;
                B.x[i] = w.x + alpha * w.p; B.r[i] = r; B.z[i] = z;
                v[0] += r * z; v[1] += r * r;
            });
            if (!qSum<2>(v, B, c, [&](const double* t) {
                    qF[1] += 1;
                    qS[S_RR] = t[1];
                    qS[S_BETA] = t[0] / qS[S_RZ];
                    qS[S_RZ] = t[0];
                    if (t[1] < qS[S_THR]) qF[0] = 1;
                    if (!(t[1] == t[1])) { qF[0] = 1; qF[2] = 1; }
                }))
                return;
        }
        it++;
    }
    if (!qBarrier(B, c)) return;
    {
        double v[1] = {0.0};
        forRows(B, rs, [&](int i, int len) {
            double r = B.b[i] - qRow(B, B.x, i, len);
            v[0] += r * r;
        });
        qSum<1>(v, B, c, [&](const double* t) { qS[S_RR] = t[0]; });
    }
    qStore(B, qL);
}

// Plain FP64 Jacobi-PCG with shared-memory vectors: the same method, rows and stopping
// rule as k_cg_solve, with r, p and Ap of each block's rows (24 bytes per row) in shared
// memory (slot m BS + t for the m-th row of thread t); x, the inverse diagonal and z (gathered
// through the matrix columns) stay in global memory.
#define OWN64_CAPMAX OWN64_CAP_ROWS   // slots per block: 3 x 8448 x 8 B = 198 KB of shared memory
__global__ void __launch_bounds__(QBC, 1) k_cg_own(Dev d, PpeBuffers B, double tol, int maxIter, int cap) {
    __shared__ QLocal qL;   // this block's copy of the solver scalars and flags
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    extern __shared__ __align__(128) unsigned char dynSmem[];
    double* const sr = reinterpret_cast<double*>(dynSmem);
    double* const sp = sr + cap;
    double* const sap = sp + cap;
    const int n = liveN(d);
    const RowSet rs = rowSet(n, QBC);   // this thread's rows (rowCount(rs) * QBC <= cap)
    QCtl c = {0u};
    {
        double v[3] = {0.0, 0.0, 0.0};
        forRowsL(B, rs, [&](int l, int i, int len) {
            const double di = 1.0 / __ldg(B.diag + i);
            const double bi = B.b[i];
            const double r = bi - qRow(B, B.x, i, len);
            const double z = r * di;
            B.dinv[i] = di; sr[l] = r; B.z[i] = z;
            v[0] += r * z; v[1] += r * r; v[2] += bi * bi;
        });
        if (!qSum<3>(v, B, c, [&](const double* t) {
                qS[S_RZ] = t[0]; qS[S_RR] = t[1]; qS[S_BB] = t[2];
                double thr = tol * tol * t[2];
                if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
                qS[S_THR] = thr;
                qS[S_SCALE] = sqrt(t[1] / (t[2] > 0 ? t[2] : 1.0));
                qF[0] = (t[2] == 0.0 || t[1] < thr) ? 1 : 0;
                qF[1] = 0;
                if (!(t[0] == t[0]) || !(t[1] == t[1])) { qF[0] = 1; qF[2] = 1; }
            }))
            return;
    }
    int it = 0;
    while (!vi(qF) && it < maxIter) {
        {   // Ap = A z + beta Ap, p = z + beta p, p.Ap
            const double beta = it ? vd(qS + S_BETA) : 0.0;
            double v[1] = {0.0};
            forRowsL(B, rs, [&](int l, int i, int len) {
                const double q = qRow(B, B.z, i, len);
                const double z = B.z[i];
                const double ap = it ? q + beta * sap[l] : q;
                const double p = it ? z + beta * sp[l] : z;
                sap[l] = ap; sp[l] = p;
                v[0] += p * ap;
            });
            if (!qSumD<1>(v, B, c, [&](const double* t) { qS[S_PAP] = t[0]; qS[S_ALPHA] = qS[S_RZ] / t[0]; }))
                return;
        }
        {   // x += alpha p, r -= alpha Ap, z = M^-1 r; r.z, r.r
            const double alpha = vd(qS + S_ALPHA);
            double v[2] = {0.0, 0.0};
            const int cnt = rowCount(rs);
            for (int m0 = 0; m0 < cnt; m0 += 4) {
                double mi[4], xo[4];
                int ii[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    ii[u] = (m0 + u < cnt) ? rowAt(rs, m0 + u) : -1;
                    mi[u] = (ii[u] >= 0) ? B.dinv[ii[u]] : 0.0;
                    xo[u] = (ii[u] >= 0) ? B.x[ii[u]] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (ii[u] < 0) continue;
                    const int l = (m0 + u) * (int)blockDim.x + (int)threadIdx.x;
                    const double r = sr[l] - alpha * sap[l];
                    const double z = r * mi[u];
                    B.x[ii[u]] = xo[u] + alpha * sp[l];
                    sr[l] = r;
                    B.z[ii[u]] = z;
                    v[0] += r * z; v[1] += r * r;
                }
            }
            if (!qSumD<2>(v, B, c, [&](const double* t) {
                    qF[1] += 1;
                    qS[S_RR] = t[1];
                    qS[S_BETA] = t[0] / qS[S_RZ];
                    qS[S_RZ] = t[0];
                    if (t[1] < qS[S_THR]) qF[0] = 1;
                    if (!(t[1] == t[1])) { qF[0] = 1; qF[2] = 1; }
                }))
                return;
        }
        it++;
    }
    if (!qBarrier(B, c)) return;
    {   // FP64 residual of the result
        double v[1] = {0.0};
        forRows(B, rs, [&](int i, int len) {
            const double r = B.b[i] - qRow(B, B.x, i, len);
            v[0] += r * r;
        });
        qSum<1>(v, B, c, [&](const double* t) { qS[S_RR] = t[0]; });
    }
    qStore(B, qL);
}

// ------------------------------------------------------------------ resident matrices
// The solvers of systems with at most one row per thread of the grid (152 x RBS = 116,736
// rows): L lanes (4, 2 or 1: as many as fit) share a row, lane l holding the entries l,
// l + L, ..., and the first `cap` entries of every lane stay in the block's shared memory from the
// first iteration to the last (slot e RBS + thread), the others, if any, are streamed.  A
// row's vector elements are registers of its lanes.  An iteration then reads nothing but z, in
// one trip to the L2 for all entries of a lane, where the streaming kernels take two dependent
// trips per eight entries; below a few thousand rows per SM these latencies and the grid
// sums are the whole time.  More than four lanes would lengthen the FP64 solver: its vector
// operations cost a warp the same for one row as for 32.
// Whole solves per step, k_cg_own / k_mx_own before and now: plain FP64 CG at 2,000 rows (27
// iterations) 0.355 -> 0.242 ms, at 6,912 (25) 0.391 -> 0.252 ms, mixed solver to 1e-10 at
// 108,000 rows (39 iterations, 1.75 refinements) 0.65 -> 0.38 ms.  Above one row per
// thread, or with long rows (resLanes), the matrix of a block no longer fits: k_cg_own and
// k_mx_own stream it.
#define RBS 768
#define RES_CAP32 36   // entries per lane: 36 x 768 x 8 B = 216 KB
#define RES_CAP64 24   // 24 x 768 x 12 B = 216 KB

struct ResRow {
    int i, l, L, len;   // row (-1: none), lane of the row, lanes per row, entries of the row
    int most;           // entries of the busiest lane of the warp
    bool any;           // the warp has a row
    size_t base, stride;
};
__device__ __forceinline__ ResRow resRow(const PpeBuffers& B, int n, int L) {
    ResRow r;
    const int G = gridDim.x, R = (n + G - 1) / G, g = threadIdx.x / L;
    r.L = L;
    r.l = threadIdx.x & (L - 1);
    const int i = blockIdx.x * R + g;
    r.i = (g < R && i < n) ? i : -1;
    r.len = r.i >= 0 ? __ldg(B.rowLen + r.i) : 0;
    r.any = __any_sync(0xffffffffu, r.i >= 0);
    r.most = __reduce_max_sync(0xffffffffu, (r.len - r.l + L - 1) / L);
    r.base = r.i >= 0 ? ellBase(B, r.i) : 0;
    r.stride = B.ellStride;
    return r;
}
// Sum of the row's off-diagonal products with x over all its lanes (the same in each): lane
// entries [0, cap) from shared memory (sc, sv), the others from the ELL arrays.
template <class T>
__device__ __forceinline__ T resDot(const ResRow& r, const int* sc, const T* sv, int cap, const int* col, const T* val,
                                    const T* x) {
    T a[4] = {T(0), T(0), T(0), T(0)};
    const int held = (min(r.most, cap) + 3) & ~3;   // cap is a multiple of 4; slots past a row's end hold zeros
    int e = 0;
    for (; e + 8 <= held; e += 8) {
        int c[8];
        T v[8], g[8];
#pragma unroll
        for (int u = 0; u < 8; u++) { c[u] = sc[(e + u) * RBS + threadIdx.x]; v[u] = sv[(e + u) * RBS + threadIdx.x]; }
#pragma unroll
        for (int u = 0; u < 8; u++) g[u] = x[c[u]];
#pragma unroll
        for (int u = 0; u < 8; u++) a[u & 3] += v[u] * g[u];
    }
    if (e < held) {
        int c[4];
        T v[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; u++) { c[u] = sc[(e + u) * RBS + threadIdx.x]; v[u] = sv[(e + u) * RBS + threadIdx.x]; }
#pragma unroll
        for (int u = 0; u < 4; u++) g[u] = x[c[u]];
#pragma unroll
        for (int u = 0; u < 4; u++) a[u] += v[u] * g[u];
        e += 4;
    }
    for (; e < r.most; e += 4) {
        int c[4];
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = r.l + (e + u) * r.L;
            const bool ok = k < r.len;
            c[u] = ok ? ldStream(col + r.base + (size_t)k * r.stride) : -1;
            v[u] = ok ? ldStream(val + r.base + (size_t)k * r.stride) : T(0);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (c[u] >= 0) a[u] += v[u] * x[c[u]];
    }
    T s = (a[0] + a[1]) + (a[2] + a[3]);
    for (int o = r.L >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}
template <class T>
__device__ __forceinline__ void resLoad(const ResRow& r, int* sc, T* sv, int cap, const int* col, const T* val) {
    const int held = min((r.most + 3) & ~3, cap);
    for (int e = 0; e < held; e++) {
        const int k = r.l + e * r.L;
        const bool ok = k < r.len;
        sc[e * RBS + threadIdx.x] = ok ? ldStream(col + r.base + (size_t)k * r.stride) : max(r.i, 0);
        sv[e * RBS + threadIdx.x] = ok ? ldStream(val + r.base + (size_t)k * r.stride) : T(0);
    }
}

// Plain FP64 Jacobi-PCG with one reduction an iteration (Chronopoulos and Gear, s-step methods,
// J. Comput. Appl. Math. 25, 1989): with q = A z,
//   gamma = r.z, delta = z.q, rho = r.r;  beta = gamma / gamma_old,
//   p.Ap = delta - beta^2 (p.Ap)_old,  alpha = gamma / p.Ap,
//   p = z + beta p,  Ap = q + beta Ap,  x += alpha p,  r -= alpha Ap,  z = M^-1 r,
// the vectors of k_cg_own, whose p.Ap comes by linearity too; the second synchronisation of an
// iteration is then a barrier (z is complete) without a sum.  The sums and the FP64 step scalars
// are k_cg_own's: no product of two sums is formed, so the right-hand side may have any scale
// that the sums themselves hold.  Stopping rule and reports of k_cg_own.
__global__ void __launch_bounds__(RBS, 1) k_cg_res(Dev d, PpeBuffers B, double tol, int maxIter, int L, int cap) {
    __shared__ QLocal qL;
    __shared__ struct { double alpha, beta, gamma, pap; int stop; } S;
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    extern __shared__ __align__(128) unsigned char dynSmem[];
    double* const sv = reinterpret_cast<double*>(dynSmem);
    int* const sc = reinterpret_cast<int*>(sv + (size_t)cap * RBS);
    const ResRow R = resRow(B, liveN(d), L);
    const bool own = R.i >= 0 && R.l == 0;
    QCtl c = {0u};
    resLoad(R, sc, sv, cap, B.col, B.val);
    double x = 0.0, r = 0.0, z = 0.0, p = 0.0, ap = 0.0, di = 0.0, dg = 0.0;
    {
        double v[3] = {0.0, 0.0, 0.0};
        if (R.any) {
            const double q = resDot<double>(R, sc, sv, cap, B.col, B.val, B.x);
            if (R.i >= 0) {
                dg = __ldg(B.diag + R.i);
                di = 1.0 / dg;
                x = B.x[R.i];
                const double bi = B.b[R.i];
                r = bi - (dg * x + q);
                z = r * di;
                if (own) {
                    B.z[R.i] = z;
                    v[0] = r * r; v[1] = bi * bi; v[2] = r * z;
                }
            }
        }
        if (!qSum<3>(v, B, c, [&](const double* t) {   // and z is complete
                qS[S_RR] = t[0]; qS[S_BB] = t[1];
                double thr = tol * tol * t[1];
                if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
                qS[S_THR] = thr;
                qS[S_SCALE] = sqrt(t[0] / (t[1] > 0 ? t[1] : 1.0));
                qF[0] = (t[1] == 0.0 || t[0] < thr) ? 1 : 0;
                qF[1] = 0;
                if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
                S.gamma = t[2];
                S.stop = qF[0] || maxIter <= 0;
            }))
            return;
    }
    while (!*(volatile int*)&S.stop) {
        double v[3] = {0.0, 0.0, 0.0}, q = 0.0;
        if (R.any) {
            q = dg * z + resDot<double>(R, sc, sv, cap, B.col, B.val, B.z);
            if (own) { v[0] = r * z; v[1] = z * q; v[2] = r * r; }
        }
        if (!qSumD<3>(v, B, c, [&](const double* t) {
                const double gamma = qF[1] ? t[0] : S.gamma, rr = qF[1] ? t[2] : qS[S_RR];   // first: of the set-up
                qS[S_RR] = rr;
                if (rr < qS[S_THR]) qF[0] = 1;
                if (!(rr == rr) || !(gamma == gamma)) { qF[0] = 1; qF[2] = 1; }
                S.stop = qF[0] || qF[1] >= maxIter;
                if (S.stop) return;
                S.beta = qF[1] ? gamma / S.gamma : 0.0;
                S.pap = qF[1] ? t[1] - S.beta * (S.beta * S.pap) : t[1];
                S.alpha = gamma / S.pap;
                S.gamma = gamma;
                qF[1] += 1;
            }, R.any))
            return;
        if (*(volatile int*)&S.stop) break;
        if (R.any) {
            const double alpha = vd(&S.alpha), beta = vd(&S.beta);
            p = z + beta * p;
            ap = q + beta * ap;
            x += alpha * p;
            r -= alpha * ap;
            z = r * di;
            if (own) B.z[R.i] = z;
        }
        if (!qBarrier(B, c)) return;
    }
    if (own) B.x[R.i] = x;
    if (!qBarrier(B, c)) return;
    {   // FP64 residual of the result
        double v[1] = {0.0};
        if (R.any) {
            const double q = resDot<double>(R, sc, sv, cap, B.col, B.val, B.x);
            if (own) {
                const double t = B.b[R.i] - (dg * x + q);
                v[0] = t * t;
            }
        }
        qSum<1>(v, B, c, [&](const double* t) { qS[S_RR] = t[0]; });
    }
    qStore(B, qL);
}

// ------------------------------------------------------------------ one cluster
// The plain FP64 solver of systems of a few thousand rows by one cluster of 16 blocks, one row
// per thread.  At that size an iteration over the whole grid is its two grid sums (arrival
// counter, poll and partials: three trips to the L2 each); inside a cluster a barrier and the
// exchange of partials stay in distributed shared memory, every block keeps its own copy of z
// (an owner writes its element into all 16), and the matrix stays in shared memory with 16-bit
// columns.  One reduction an iteration (Chronopoulos and Gear, s-step methods, J. Comput. Appl.
// Math. 25, 1989): with q = A z,
//   gamma = r.z, delta = z.q, rho = r.r;  beta = gamma / gamma_old,
//   p.Ap = delta - beta^2 (p.Ap)_old,  alpha = gamma / p.Ap,
//   p = z + beta p,  Ap = q + beta Ap,  x += alpha p,  r -= alpha Ap,  z = M^-1 r,
// the same vectors as k_cg_res, whose p.Ap it forms by linearity too, and like there the set-up's
// sums, the step scalars and the residual of the result are FP64.  The first warp has no
// rows: it sums the warps' partials and forms the step scalars.
// Bound by latency: at the 2-D dam's 2,916 rows an iteration takes ~9,600 cycles, the product 1,700,
// delta and its barrier 1,900, collecting the partials 750, the FP64 scalars 2,000, the update
// with the next sums 2,500.  Only delta waits for the product, so z is
// published as soon as it is known, and the x update and the trees of the next iteration's r.z
// and r.r run between arrival and wait of its barrier (three sums after the product, all in one
// exchange, took 18% longer).
#define CLB 16                 // blocks of the cluster
#define CL_ROWS 256            // rows of a block at most
struct ClShared {
    // the warps' partials (every warp writes its own into all blocks), two sets in turn
    float2 part[2][3][CL_ROWS / 32][CLB];
    double alpha, beta;
    int stop;
};
__device__ __forceinline__ void clArrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void clWait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned clAddr(const void* p, unsigned rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void clStore(const void* p, unsigned rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(clAddr(p, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ void clStore(const void* p, unsigned rank, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(clAddr(p, rank)), "f"(v.x), "f"(v.y) : "memory");
}
// Sums over the cluster, in float-float from the warp level on (as qSumD): every warp with rows
// writes its partial of value q into set `set` of all blocks (clPush); after a cluster barrier the
// first warp of each block sums the partials in the same order (clTotal, in every lane).
// NV values, v[k] as value q0 + k dq; their trees run side by side.
template <int NV>
__device__ __forceinline__ void clPush(const double (&v)[NV], int q0, int dq, int set, ClShared& S, unsigned rank) {
    const int lane = threadIdx.x & 31, w = ((int)threadIdx.x >> 5) - 1;
    df a[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) a[k] = dfD(v[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) a[k] += shflXorDF(a[k], o);
    if (lane < CLB)
#pragma unroll
        for (int k = 0; k < NV; k++) clStore(&S.part[set][q0 + k * dq][w][rank], lane, make_float2(a[k].h, a[k].l));
}
// The same in FP64, for the sums of the set-up and of the result.
template <int NV>
__device__ __forceinline__ void clPushD(double (&v)[NV], int set, ClShared& S, unsigned rank) {
    const int lane = threadIdx.x & 31, w = ((int)threadIdx.x >> 5) - 1;
#pragma unroll
    for (int q = 0; q < NV; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if (lane < CLB) clStore(&S.part[set][q][w][rank], lane, v[q]);
    }
}
template <int NV>
__device__ __forceinline__ void clTotalD(int set, const ClShared& S, double (&a)[NV]) {
    const int lane = threadIdx.x & 31, nw = ((int)blockDim.x >> 5) - 1;
#pragma unroll
    for (int q = 0; q < NV; q++) {
        a[q] = 0.0;
        for (int m = lane; m < nw * CLB; m += 32) {
            const float2 x = S.part[set][q][0][m];   // an FP64 value's two words
            a[q] += __hiloint2double(__float_as_int(x.y), __float_as_int(x.x));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
    }
}
template <int NV>
__device__ __forceinline__ void clTotal(int set, const ClShared& S, df (&a)[NV]) {
    const int lane = threadIdx.x & 31, nw = ((int)blockDim.x >> 5) - 1;
#pragma unroll
    for (int q = 0; q < NV; q++) a[q] = dfF(0.f);
    for (int m = lane; m < nw * CLB; m += 32)
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const float2 x = S.part[set][q][0][m];
            a[q] += df{x.x, x.y};
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NV; q++) a[q] += shflXorDF(a[q], o);
}
__global__ void __launch_bounds__(CL_ROWS + 32, 1) k_cg_cluster(Dev d, PpeBuffers B, double tol, int maxIter, int cap) {
    __shared__ QLocal qL;
    __shared__ ClShared S;
    extern __shared__ __align__(128) unsigned char dynSmem[];
    double* const zc = reinterpret_cast<double*>(dynSmem);
    const int n = liveN(d), T = (int)blockDim.x - 32;
    double* const sv = zc + CLB * T;
    unsigned short* const sc = reinterpret_cast<unsigned short*>(sv + (size_t)cap * T);
    unsigned rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    // a block's shared memory may be written by another only once it has started: arrive here, wait
    // before the first push, the matrix loads between the two
    clArrive();
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    const int t = (int)threadIdx.x - 32;                                  // row of the block, negative: none
    const int i = t >= 0 && (int)rank * T + t < n ? (int)rank * T + t : -1;
    const bool own = i >= 0;
    const int len = own ? __ldg(B.rowLen + i) : 0;
    const int most = __reduce_max_sync(0xffffffffu, len);
    const size_t base = own ? ellBase(B, i) : 0;
    const int held = min(most, cap);
    if (t >= 0)
#pragma unroll 8
        for (int e = 0; e < held; e++) {
            const bool ok = e < len;
            sc[e * T + t] = ok ? (unsigned short)ldStream(B.col + base + (size_t)e * B.ellStride) : (unsigned short)0;
            sv[e * T + t] = ok ? ldStream(B.val + base + (size_t)e * B.ellStride) : 0.0;
        }
    for (int k = threadIdx.x; k < n; k += blockDim.x) zc[k] = B.x[k];
    __syncthreads();
    double dg = 1.0, x = 0.0, r = 0.0, z = 0.0, p = 0.0, ap = 0.0, di = 1.0, bi = 0.0;
    // (A v)_i of the vector in zc, v its own element
    auto product = [&](double v) {
        double a[2] = {dg * v, 0.0};   // (an FP64 operation of a warp takes 64 issue slots: few sums, no padding)
        int e = 0;
        for (; e + 4 <= held; e += 4) {
            double g[4];
#pragma unroll
            for (int u = 0; u < 4; u++) g[u] = zc[sc[(e + u) * T + t]];
#pragma unroll
            for (int u = 0; u < 4; u++) a[u & 1] += sv[(e + u) * T + t] * g[u];
        }
        for (; e < held; e++) a[e & 1] += sv[e * T + t] * zc[sc[e * T + t]];
        for (; e < len; e++)
            a[0] += ldStream(B.val + base + (size_t)e * B.ellStride) * zc[ldStream(B.col + base + (size_t)e * B.ellStride)];
        return a[0] + a[1];
    };
    auto publish = [&](double v) {   // into every block's copy
#pragma unroll
        for (unsigned q = 0; q < CLB; q++) clStore(zc + i, q, v);
    };
    if (own) {
        dg = __ldg(B.diag + i);
        di = 1.0 / dg;
        x = B.x[i];
        bi = B.b[i];
        r = bi - product(x);
        z = r * di;
    }
    clWait();   // every block of the cluster has started
    if (t >= 0) {
        double v[3] = {bi * bi, r * r, r * z};
        clPushD<3>(v, 0, S, rank);
    }
    clArrive();
    clWait();   // also ends every block's reads of x
    double gamma = 0.0, pap = 0.0, invGamma = 0.0;   // thread 0 (invGamma: 1 / gamma, 0 before the first iteration)
    if (threadIdx.x < 32) {
        double a[3];
        clTotalD<3>(0, S, a);
        if (threadIdx.x == 0) {
            const double bb = a[0], rr = a[1];
            gamma = a[2];
            qS[S_BB] = bb;
            double thr = tol * tol * bb;
            if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
            qS[S_THR] = thr;
            qS[S_RR] = rr;
            qS[S_SCALE] = sqrt(rr / (bb > 0 ? bb : 1.0));
            qF[0] = (bb == 0.0 || rr < thr) ? 1 : 0;
            qF[1] = 0;
            if (!(rr == rr)) { qF[0] = 1; qF[2] = 1; }
            S.stop = qF[0] || maxIter <= 0;
        }
    }
    if (own) publish(z);
    if (t >= 0) {   // gamma and rho of the first iteration
        const double v[2] = {r * z, r * r};
        clPush<2>(v, 0, 2, 1, S, rank);
    }
    clArrive();
    clWait();
    for (int set = 1; !S.stop; set ^= 1) {
        double q = 0.0;
        if (own) q = product(z);
        if (t >= 0) {
            const double v[1] = {own ? z * q : 0.0};
            clPush<1>(v, 1, 0, set, S, rank);
        }
        clArrive();
        clWait();
        if (threadIdx.x < 32) {
            df a[3];
            clTotal<3>(set, S, a);
            if (threadIdx.x == 0) {
                const double g = qF[1] ? dD(a[0]) : gamma, rr = qF[1] ? dD(a[2]) : qS[S_RR];   // first: of the set-up
                // g / gamma by the reciprocal taken while the other blocks arrived, and its remainder (a
                // division here would be a tenth of the iteration)
                double beta = g * invGamma;
                beta = fma(fma(-beta, gamma, g), invGamma, beta);
                pap = dD(a[1]) - beta * (beta * pap);
                gamma = g;
                S.alpha = g / pap;
                S.beta = beta;
                if (rr < qS[S_THR]) qF[0] = 1;
                if (!(rr == rr) || !(g == g)) { qF[0] = 1; qF[2] = 1; }
                S.stop = qF[0] || qF[1] >= maxIter;
                if (S.stop) qS[S_RR] = rr;
            }
        }
        __syncthreads();
        if (S.stop) break;
        if (own) {
            const double alpha = S.alpha, beta = S.beta;
            p = z + beta * p;
            ap = q + beta * ap;
            r -= alpha * ap;
            z = r * di;
            publish(z);
        }
        clArrive();   // z is published; the rest runs while the other blocks arrive
        if (own) x += S.alpha * p;
        if (t >= 0) {
            const double v[2] = {own ? r * z : 0.0, own ? r * r : 0.0};
            clPush<2>(v, 0, 2, set ^ 1, S, rank);
        }
        if (threadIdx.x == 0) {
            qF[1] += 1;
            invGamma = 1.0 / gamma;
        }
        clWait();
    }
    // FP64 residual of the result
    clArrive();
    clWait();   // every block has left its last product
    if (own) { B.x[i] = x; publish(x); }
    clArrive();
    clWait();
    if (t >= 0) {
        const double e = own ? bi - product(x) : 0.0;
        double v[1] = {e * e};
        clPushD<1>(v, 0, S, rank);
    }
    clArrive();
    clWait();
    if (threadIdx.x < 32) {
        double a[1];
        clTotalD<1>(0, S, a);
        if (threadIdx.x == 0) qS[S_RR] = a[0];
    }
    __syncthreads();
    if (rank == 0) qStore(B, qL);
}
// Shared memory of k_cg_cluster for a system of `rows` rows (T threads with rows per block, cap
// entries of each held), 0 where a block's part does not fit.
static size_t clusterShape(const PpeBuffers& B, int rows, int* T, int* cap) {
    *T = ((rows + CLB - 1) / CLB + 31) / 32 * 32;
    if (rows <= 0 || *T > CL_ROWS) return 0;
    const size_t room = 220 * 1024 - (size_t)CLB * *T * 8;
    *cap = std::min((B.K + 3) / 4 * 4, (int)(room / ((size_t)*T * 10)) / 4 * 4);
    return (size_t)CLB * *T * 8 + (size_t)*cap * *T * 10;
}
static cudaError_t launchCluster(const Dev& d, const PpeBuffers& B, double tol, int maxIter, int T, int cap, size_t dyn,
                                 cudaStream_t s) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(CLB);
    c.blockDim = dim3(T + 32);
    c.dynamicSmemBytes = dyn;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CLB; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k_cg_cluster, d, B, tol, maxIter, cap);
}
// 1 when this GPU can hold a cluster of the largest shape.
static int clusterAvailable() {
    if (cudaFuncSetAttribute(k_cg_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(k_cg_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(CLB);
    c.blockDim = dim3(CL_ROWS + 32);
    c.dynamicSmemBytes = 220 * 1024;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CLB; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_cg_cluster, &c) != cudaSuccess) { cudaGetLastError(); return 0; }
    return clusters > 0;
}

// Mixed FP32/FP64 solver: method, stopping rules and reports of k_mx_own (LEARNED as there:
// the residual of the start is in B.r, its correction and their product in B.cdir and B.cq).
template <bool LEARNED>
__global__ void __launch_bounds__(RBS, 1) k_mx_res(Dev d, PpeBuffers B, double tol, int maxIter, double eta2, int L, int cap) {
    __shared__ QLocal qL;
    __shared__ df rz, stop2;   // inner solve: r.z, and the squared residual norm that ends it
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    extern __shared__ __align__(128) unsigned char dynSmem[];
    float* const sv = reinterpret_cast<float*>(dynSmem);
    int* const sc = reinterpret_cast<int*>(sv + (size_t)cap * RBS);
    const ResRow R = resRow(B, liveN(d), L);
    const bool own = R.i >= 0 && R.l == 0;
    QCtl c = {0u};
    resLoad(R, sc, sv, cap, B.col, B.valf);
    // FP64 residual of B.x, whose element of the row is x
    double x = 0.0, r = 0.0;
    auto residual = [&]() {
        const double q = resDot<double>(R, nullptr, nullptr, 0, B.col, B.val, B.x);
        return R.i >= 0 ? B.b[R.i] - (__ldg(B.diag + R.i) * x + q) : 0.0;
    };
    float dgf = 0.f, dif = 0.f;
    {
        double v[LEARNED ? 4 : 2] = {};
        if (R.any) {
            if (R.i >= 0) { x = B.x[R.i]; dgf = __ldg(B.diagf + R.i); dif = __ldg(B.diagInvf + R.i); }
            if (LEARNED) r = R.i >= 0 ? B.r[R.i] : 0.0;
            else r = residual();
            if (own) {
                const double bi = B.b[R.i];
                v[0] = r * r;
                v[1] = bi * bi;
                if (LEARNED) {
                    const double q = (double)__ldg(B.cq + R.i);
                    v[LEARNED ? 2 : 0] = r * q;
                    v[LEARNED ? 3 : 0] = q * q;
                }
            }
        }
        if (!qSum<LEARNED ? 4 : 2>(v, B, c, [&](const double* t) { mxStart<LEARNED>(qL, t, tol, eta2); })) return;
        if (LEARNED) {
            const double th = vd(qS + S_OMEGA);
            if (R.i >= 0 && th != 0.0) {
                x += th * (double)__ldg(B.cdir + R.i);
                r -= th * (double)__ldg(B.cq + R.i);
                if (own) B.x[R.i] = x;
            }
        }
    }
    int total = 0, refine = 0;
    while (!vi(qF) && total < maxIter && refine <= 20) {
        float xf = 0.f, rf = 0.f, zf = 0.f, pf = 0.f, apf = 0.f;
        {   // inner start: r_f = r / ||r||, z = M^-1 r_f, x_f = 0
            df a[2] = {dfF(0.f), dfF(0.f)};
            if (R.any) {
                rf = (float)(r * vd(qS + S_INV));
                zf = rf * dif;
                if (own) {
                    B.zf[R.i] = zf;
                    a[0] = prod2(rf, zf);
                    a[1] = prod2(rf, rf);
                }
            }
            if (!qSumF2<2>(a, B, c, [&](const df* t) {
                    rz = t[0];
                    stop2 = dfD(dD(t[1]) * qS[S_ETA2]);
                    qF[3] = 0;
                }))
                return;
        }
        int inner = 0;
        while (true) {
            {   // Ap = A z + beta Ap, p = z + beta p, p.Ap
                df a[1] = {dfF(0.f)};
                if (R.any) {
                    const float beta = inner ? vf(qL.scalf + SF_BETA) : 0.f;
                    const float q = dgf * zf + resDot<float>(R, sc, sv, cap, B.col, B.valf, B.zf);
                    apf = inner ? q + beta * apf : q;
                    pf = inner ? zf + beta * pf : zf;
                    if (own) a[0] = prod2(pf, apf);
                }
                if (!qSumF2<1>(a, B, c, [&](const df* t) { qL.scalf[SF_ALPHA] = divF(rz, t[0]); }, R.any)) return;
            }
            {   // x_f += alpha p, r -= alpha Ap, z = M^-1 r; r.z, r.r
                const float alpha = vf(qL.scalf + SF_ALPHA);
                df a[2] = {dfF(0.f), dfF(0.f)};
                xf += alpha * pf;
                rf -= alpha * apf;
                zf = rf * dif;
                if (own) {
                    B.zf[R.i] = zf;
                    a[0] = prod2(rf, zf);
                    a[1] = prod2(rf, rf);
                }
                if (!qSumF2<2>(a, B, c, [&](const df* t) {
                        qF[1] += 1;
                        qL.scalf[SF_BETA] = divF(t[0], rz);
                        rz = t[0];
                        if (t[1] < stop2 || !(t[1].h == t[1].h)) qF[3] = 1;
                    }, R.any))
                    return;
            }
            inner++;
            if (vi(qF + 3) || total + inner >= maxIter || inner >= 400) break;
        }
        total += inner;
        {   // x += ||r|| x_f (FP64), then the FP64 residual r = b - A x
            if (R.any) x += vd(qS + S_SQRT) * (double)xf;
            if (own) B.x[R.i] = x;
            if (!qBarrier(B, c)) return;
            double v[1] = {0.0};
            if (R.any) {
                r = residual();
                if (own) v[0] = r * r;
            }
            if (!qSum<1>(v, B, c, [&](const double* t) {
                    qS[S_RR] = t[0];
                    qS[S_SQRT] = sqrt(t[0]);
                    qS[S_INV] = 1.0 / sqrt(t[0]);
                    qS[S_ETA2] = fmax(eta2, 0.25 * qS[S_THR] / t[0]);
                    if (t[0] < qS[S_THR]) qF[0] = 1;
                    if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
                    qF[4] += 1;
                }))
                return;
        }
        refine++;
    }
    qStore(B, qL);
}

// Jacobi-preconditioned BiCGSTAB (solver_type 1: Eigen::BiCGSTAB, src/MpsPressure.cpp:448-468;
// van der Vorst 1992 with the preconditioner on the right), in one cooperative launch: per
// iteration two SpMVs and five grid synchronisations (y and z must be complete before their
// SpMVs; (r0, v), (t, t) and (t, s), (r, r) and (r0, r) are grid sums).  The shadow residual
// is restarted when (r0, r) vanishes relative to its start, the stopping rule is
// ||r||^2 < tol^2 ||b||^2 on the recurrence residual, and the FP64 residual of the result is
// reported.
__global__ void __launch_bounds__(QBC, 1) k_bicgstab(Dev d, PpeBuffers B, double tol, int maxIter) {
    __shared__ QLocal qL;   // this block's copy of the solver scalars and flags
    qInit(qL);
    double* const qS = qL.scal;
    int* const qF = qL.flag;
    const int n = liveN(d);
    const RowSet rs = rowSet(n, QBC);   // this thread's rows
    QCtl c = {0u};
    double *r0 = B.bs[0], *sv = B.bs[1], *zz = B.bs[2], *tv = B.bs[3], *y = B.z, *v = B.Ap;
    auto restart = [&](bool first) -> bool {
        double a[2] = {0.0, 0.0};
        forRows(B, rs, [&](int i, int len) {
            if (first) B.dinv[i] = 1.0 / __ldg(B.diag + i);
            double r = B.b[i] - qRow(B, B.x, i, len);
            B.r[i] = r; r0[i] = r; B.p[i] = 0.0; v[i] = 0.0;
            a[0] += r * r;
            if (first) a[1] += B.b[i] * B.b[i];
        });
        return qSum<2>(a, B, c, [&](const double* t) {
            if (first) {
                qS[S_BB] = t[1];
                double thr = tol * tol * t[1];
                if (thr < 2.2250738585072014e-308) thr = 2.2250738585072014e-308;
                qS[S_THR] = thr;
                qS[S_SCALE] = sqrt(t[0] / (t[1] > 0 ? t[1] : 1.0));
                qF[1] = 0;
                if (t[1] == 0.0) qF[0] = 1;
            }
            qS[S_RR] = qS[S_RHO] = qS[S_R0N2] = t[0];
            qS[S_RHOOLD] = qS[S_ALPHA] = qS[S_OMEGA] = 1.0;
            qF[5] = 0;
            if (t[0] < qS[S_THR]) qF[0] = 1;
            if (!(t[0] == t[0])) { qF[0] = 1; qF[2] = 1; }
        });
    };
    if (!restart(true)) return;
    int it = 0;
    while (!vi(qF) && it < maxIter) {
        {   // p = r + beta (p - w v), y = M^-1 p
            const double rho = vd(qS + S_RHO), w = vd(qS + S_OMEGA);
            const double beta = (rho / vd(qS + S_RHOOLD)) * (vd(qS + S_ALPHA) / w);
            forOwn(rs, [&](int i) {
                double p = B.r[i] + beta * (B.p[i] - w * v[i]);
                B.p[i] = p;
                y[i] = p * B.dinv[i];
            });
            if (!qBarrier(B, c)) return;
        }
        {   // v = A y, alpha = rho / (r0, v)
            double a[1] = {0.0};
            forRows(B, rs, [&](int i, int len) {
                double q = qRow(B, y, i, len);
                v[i] = q;
                a[0] += r0[i] * q;
            });
            if (!qSum<1>(a, B, c, [&](const double* t) {
                    double al = qS[S_RHO] / t[0];
                    qS[S_ALPHA] = al;
                    if (!(al == al) || t[0] == 0.0) { qF[0] = 1; qF[2] = 1; }
                }))
                return;
        }
        if (vi(qF)) break;
        {   // s = r - alpha v, z = M^-1 s
            const double alpha = vd(qS + S_ALPHA);
            forOwn(rs, [&](int i) {
                double s = B.r[i] - alpha * v[i];
                sv[i] = s;
                zz[i] = s * B.dinv[i];
            });
            if (!qBarrier(B, c)) return;
        }
        {   // t = A z, w = (t, s) / (t, t)
            double a[2] = {0.0, 0.0};
            forRows(B, rs, [&](int i, int len) {
                double q = qRow(B, zz, i, len);
                tv[i] = q;
                a[0] += q * q;
                a[1] += q * sv[i];
            });
            if (!qSum<2>(a, B, c, [&](const double* t) { qS[S_OMEGA] = (t[0] > 0.0) ? t[1] / t[0] : 0.0; }))
                return;
        }
        {   // x += alpha y + w z, r = s - w t; (r, r) and the next rho = (r0, r)
            const double alpha = vd(qS + S_ALPHA), w = vd(qS + S_OMEGA);
            double a[2] = {0.0, 0.0};
            forOwn(rs, [&](int i) {
                B.x[i] += alpha * y[i] + w * zz[i];
                double r = sv[i] - w * tv[i];
                B.r[i] = r;
                a[0] += r * r;
                a[1] += r0[i] * r;
            });
            if (!qSum<2>(a, B, c, [&](const double* t) {
                    qF[1] += 1;
                    qS[S_RR] = t[0];
                    qS[S_RHOOLD] = qS[S_RHO];
                    qS[S_RHO] = t[1];
                    if (t[0] < qS[S_THR]) qF[0] = 1;
                    else if (fabs(t[1]) < 4.930380657631324e-32 * qS[S_R0N2]) qF[5] = 1;   // eps^2
                    if (!(t[0] == t[0]) || qS[S_OMEGA] == 0.0) { qF[0] = 1; qF[2] = 1; }
                }))
                return;
        }
        it++;
        if (vi(qF + 5) && !vi(qF))
            if (!restart(false)) return;
    }
    if (!qBarrier(B, c)) return;
    {
        double a[1] = {0.0};
        forRows(B, rs, [&](int i, int len) {
            double r = B.b[i] - qRow(B, B.x, i, len);
            a[0] += r * r;
        });
        qSum<1>(a, B, c, [&](const double* t) { qS[S_RR] = t[0]; });
    }
    qStore(B, qL);
}

// kind: 0 plain FP64, 1 mixed, 2 mixed with the matrix-free inner operator, 3 mixed with
// the compact scaled inner operator, 4 mixed with the staged tiles, 5 mixed with the
// pipelined inner CG, 6 BiCGSTAB, 7 mixed with block-owned rows (one block per SM), 8 plain
// FP64 with block-owned rows (one block per SM), 9 resident matrices (one block per SM)
int ppePersistentGrid(int kind) {
    int dev = 0, sms = 0, coop = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return 0;
    if (kind == 7) {
        for (int k = 0; k < 6; k++) {
            const void* f = ownKernel(k & 1, 2 + k / 2);
            if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, OWN_SMEM) != cudaSuccess) return 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, QBX, OWN_SMEM) != cudaSuccess || per <= 0) return 0;
        }
        return sms;   // one block per SM: the ranges are sized for it
    }
    if (kind == 8) {
        const int dyn = OWN64_CAPMAX * 24;
        if (cudaFuncSetAttribute(k_cg_own, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cg_own, QBC, dyn) != cudaSuccess || per <= 0) return 0;
        return sms;
    }
    if (kind == 10) return clusterAvailable();
    if (kind == 9) {   // resident matrices, one block per SM
        for (const void* f : {(const void*)k_cg_res, (const void*)k_mx_res<false>, (const void*)k_mx_res<true>}) {
            const int dyn = f == (const void*)k_cg_res ? RES_CAP64 * RBS * 12 : RES_CAP32 * RBS * 8;
            if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess) return 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, RBS, dyn) != cudaSuccess || per <= 0) return 0;
        }
        return sms;
    }
    if (kind == 4) {
        if (cudaFuncSetAttribute(k_mx_solve<OP_TILED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(TsSmem)) != cudaSuccess)
            return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mx_solve<OP_TILED>, QB, sizeof(TsSmem)) != cudaSuccess ||
            per <= 0)
            return 0;
        return per * sms;
    }
    cudaError_t e = kind == 6   ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_bicgstab, QBC, 0)
                    : kind == 5 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mx_pipe, QBX, 0)
                    : kind == 3 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mx_solve<OP_H16>, QBX, 0)
                    : kind == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mx_solve<OP_MATFREE>, QBX, 0)
                    : kind == 1 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mx_solve<OP_ELL32>, QBX, 0)
                                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cg_solve, QBC, 0);
    if (e != cudaSuccess || per <= 0) return 0;
    return per * sms;
}

static int finishPersistent(const PpeBuffers& B, cudaStream_t s, int* iters, int* refinements, double* relres,
                            double* relres0) {
    // one copy into page-locked memory (three into pageable variables waited for the stream three times)
    if (cudaMemcpyAsync(B.hostCtl, B.scal, PPE_CTL_BYTES, cudaMemcpyDeviceToHost, s) != cudaSuccess) return MPSGPU_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return MPSGPU_ERR_CUDA;
    const double* sc = static_cast<const double*>(B.hostCtl);
    const int* f = reinterpret_cast<const int*>(sc + 32);
    const unsigned int abortWord = *reinterpret_cast<const unsigned int*>(f + PPE_CTL_FLAGS + QB_ABT);
    if (abortWord) return MPSGPU_ERR_CUDA;   // a grid-barrier wait ran out (reported by the caller)
    *iters = f[1];
    if (refinements) *refinements = f[4];
    double bb = sc[S_BB] > 0 ? sc[S_BB] : 1.0;
    *relres = (sc[S_BB] > 0) ? sqrt(sc[S_RR] / bb) : 0.0;
    *relres0 = sc[S_SCALE];
    if (f[2] || !f[0]) return MPSGPU_ERR_NOT_CONVERGED;
    return 0;
}

// flags and barrier words (adjacent: PPE_CTL_FLAGS words of flags first)
static void qClear(const PpeBuffers& B, cudaStream_t s) {
    cudaMemsetAsync(B.flag, 0, (PPE_CTL_FLAGS + QB_WORDS) * sizeof(int), s);
}

int ppeSolveBicgstab(const Dev& d, const PpeBuffers& B, double tol, int maxIter, cudaStream_t s, int* iters,
                     double* relres, double* relres0, Prof* prof) {
    if (B.pgridBi <= 0) return MPSGPU_ERR_UNSUPPORTED;
    bool pr = prof && prof->on;
    qClear(B, s);
    Dev dd = d;
    PpeBuffers bb = B;
    double t = tol;
    int mi = maxIter;
    void* args[4] = {&dd, &bb, &t, &mi};
    if (pr) prof->begin(PROF_PPE_SOLVE, s);
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_bicgstab, B.pgridBi, QBC, args, 0, s);
    if (pr) prof->end(s);
    if (e != cudaSuccess) return MPSGPU_ERR_CUDA;
    countLaunch(1);
    return finishPersistent(B, s, iters, nullptr, relres, relres0);
}

// Rows up to which one cluster takes the plain FP64 solve, all that its blocks hold at one row per
// thread.  Three first solves of a run (65 to 76 iterations, set-up included) by k_cg_cluster and
// k_cg_res at 1,000 rows 463 / 599 us, 2,048 rows 535 / 658, 2,916 rows 567 / 682, 4,000 rows
// 650 / 713: the gain shrinks as the 16 SMs' FP64 pipes fill.
#define CLUSTER_MAX_ROWS 4096
// Lanes per row of the resident solvers: 4, 2 or 1, as many as give every row of `rows` its
// lanes in one round of the grid; 0: too many rows, or too many entries (`filled` a row in a filled
// neighbourhood, `cap` of each lane held) are left to be streamed in every product, which the
// solvers without a resident matrix do eight at a time.  Whole solves, resident / k_cg_own and
// resident / k_mx_own: 97k rows of 92 entries (6.6M and 5.4M streamed) 0.561 / 0.591 and 0.533 / 0.549 ms,
// 115k of 80 (6.5M, 5.1M) 0.670 / 0.652 and 0.509 / 0.561, 115k of 92 (7.8M, 6.5M) 0.710 / 0.646 and
// 0.603 / 0.589, 61k of 122 (6.0M, 5.2M) 0.600 / 0.597 and 0.560 / 0.570, 97k of 122 (9.5M, 8.4M) 0.698 /
// 0.657 and 0.755 / 0.627.
#define RES_STREAMED 6e6
static int resLanes(int rows, int grid, double filled, int cap) {
    for (int L = 4; L; L >>= 1)
        if (rows <= grid * (RBS / L)) return rows * (filled - (double)(L * cap)) <= RES_STREAMED ? L : 0;
    return 0;
}

int ppeSolvePersistent(const Dev& d, const PpeBuffers& B, int mixed, double tol, int maxIter, cudaStream_t s,
                       int* iters, int* refinements, double* relres, double* relres0, Prof* prof) {
    int grid = !mixed ? B.pgridCg
                      : (B.matfree == 4 ? B.pgridPipe
                                        : (B.matfree == 3 ? B.pgridTs
                                                          : (B.matfree == 2 ? B.pgridH16 : (B.matfree ? B.pgridMf : B.pgridMx))));
    if (grid <= 0) return MPSGPU_ERR_UNSUPPORTED;
    bool pr = prof && prof->on;
    qClear(B, s);
    if (mixed && !B.prepared) {
        if (pr) prof->begin(PROF_PPE_OTHER, s);
        k_mixed_prepare<<<gridFor(d.N0, 256), 256, 0, s>>>(d, B);
        if (pr) prof->end(s);
        countLaunch(1);
    }
    Dev dd = d;
    PpeBuffers bb = B;
    // inner floor 1e-6: from a good warm start one FP32 inner solve reaches the whole
    // reduction and a single FP64 refinement confirms it (measured at 864k rows: one
    // refinement instead of two, 1.86 -> 1.74 ms); a coarser floor forces extra refinements
    double t = tol, eta2 = 1e-6 * 1e-6;
    int mi = maxIter;
    void* args[6] = {&dd, &bb, &t, &mi, &eta2, nullptr};
    if (!mixed && !B.ownOff && B.cluster && d.N0 <= CLUSTER_MAX_ROWS) {
        int T = 0, cap = 0;
        const size_t dyn = clusterShape(B, d.N0, &T, &cap);
        if (dyn) {
            if (pr) prof->begin(PROF_PPE_SOLVE, s);
            const cudaError_t e = launchCluster(d, B, tol, maxIter, T, cap, dyn, s);
            if (pr) prof->end(s);
            if (e != cudaSuccess) return MPSGPU_ERR_CUDA;
            countLaunch(1);
            return finishPersistent(B, s, iters, refinements, relres, relres0);
        }
    }
    const int lanes = B.matfree == 0 && !B.ownOff && B.pgridRes > 0
                          ? resLanes(d.N0, B.pgridRes, d.P.numNeighZero, mixed ? RES_CAP32 : RES_CAP64)
                          : 0;
    if (lanes) {
        // at most one row per thread: the matrix stays in shared memory.  The rows are spread
        // over all SMs (the FP64 pipe and the latencies are per SM), 16 to a block at least
        const int need = (B.K + lanes - 1) / lanes;
        int L = lanes, cap = std::min((need + 3) / 4 * 4, mixed ? RES_CAP32 : RES_CAP64);
        const int g = std::min(B.pgridRes, (d.N0 + 15) / 16);
        void* aPlain[6] = {&dd, &bb, &t, &mi, &L, &cap};
        void* aMixed[7] = {&dd, &bb, &t, &mi, &eta2, &L, &cap};
        const void* fn = !mixed ? (const void*)k_cg_res : B.cdir ? (const void*)k_mx_res<true> : (const void*)k_mx_res<false>;
        if (pr) prof->begin(PROF_PPE_SOLVE, s);
        cudaError_t e = cudaLaunchCooperativeKernel(fn, g, RBS, mixed ? aMixed : aPlain,
                                                    (size_t)cap * RBS * (mixed ? 8 : 12), s);
        if (pr) prof->end(s);
        if (e != cudaSuccess) return MPSGPU_ERR_CUDA;
        countLaunch(1);
        return finishPersistent(B, s, iters, refinements, relres, relres0);
    }
    if (!mixed && !B.ownOff && B.pgridOwn64 > 0 && B.ownCap64 > 0) {
        // block-owned rows: r, p, Ap of each block in its shared memory
        int cap = B.ownCap64;
        void* a4[5] = {&dd, &bb, &t, &mi, &cap};
        if (pr) prof->begin(PROF_PPE_SOLVE, s);
        cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_cg_own, B.pgridOwn64, QBC, a4, (size_t)cap * 24, s);
        if (pr) prof->end(s);
        if (e != cudaSuccess) return MPSGPU_ERR_CUDA;
        countLaunch(1);
        return finishPersistent(B, s, iters, refinements, relres, relres0);
    }
    if (mixed && B.matfree == 0 && !B.ownOff && B.pgridOwn > 0 && B.ownCap > 0) {
        // block-owned rows: the FP32 inner-CG vectors of each block in its shared memory
        int cap = B.ownCap;
        args[5] = &cap;
        if (pr) prof->begin(PROF_PPE_SOLVE, s);
        cudaError_t e = cudaLaunchCooperativeKernel(ownKernel(B.cdir != nullptr, B.ownVec), B.pgridOwn, QBX, args,
                                                    (size_t)cap * 4 * B.ownVec, s);
        if (pr) prof->end(s);
        if (e != cudaSuccess) return MPSGPU_ERR_CUDA;
        countLaunch(1);
        return finishPersistent(B, s, iters, refinements, relres, relres0);
    }
    if (pr) prof->begin(PROF_PPE_SOLVE, s);
    const void* fn = !mixed              ? (const void*)k_cg_solve
                     : B.matfree == 4    ? (const void*)k_mx_pipe
                     : B.matfree == 3    ? (const void*)k_mx_solve<OP_TILED>
                     : B.matfree == 2    ? (const void*)k_mx_solve<OP_H16>
                     : B.matfree == 1    ? (const void*)k_mx_solve<OP_MATFREE>
                                         : (const void*)k_mx_solve<OP_ELL32>;
    size_t dyn = (mixed && B.matfree == 3) ? sizeof(TsSmem) : 0;
    const int bs = !mixed ? QBC : (B.matfree == 3 ? QB : QBX);
    cudaError_t e = cudaLaunchCooperativeKernel(fn, grid, bs, args, dyn, s);
    if (pr) prof->end(s);
    if (e != cudaSuccess) return MPSGPU_ERR_CUDA;
    countLaunch(1);
    return finishPersistent(B, s, iters, refinements, relres, relres0);
}
