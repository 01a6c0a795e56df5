// qms_solver.cu -- the per-step linear solve that replaces MKL PARDISO
// (3D/QMS_3D.f90:1314-1317 phase 13, F:2193-2203 phases 23/33).
//
// Structure of one solve (steady init or one backward-Euler step):
//   b, Dirichlet values of x  <- K7 (qms_exact.cu)
//   repeat (FP64 iterative refinement):
//       r = D^-1 (b - M x)                       FP64 matrix-free residual (K3)
//       stop when ||r|| <= tol * ||x||
//       e ~= (D^-1 M)^-1 r / ||r||               inner Krylov in T (FP32 = mixed, FP64 = plain)
//       x += ||r|| e                             FP64 accumulation
// Inner Krylov: PCG for the symmetric steady magnetostatic problem (v = 0, V
// block identically zero), FGMRES (or BiCGSTAB) on the row-scaled operator for
// every nonsymmetric system.  All Krylov scalars live in device memory and are
// formed from deterministic block partial sums by one-block finalize kernels or
// by the last block of a launch, so the vector kernels never wait for the
// host; the host only reads the residual estimate to decide when to stop.
#include "qms_internal.h"
#include "qms_solver.h"
#include "qms_pdl.cuh"
#include "qms_pl.h"

#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

// --------------------------------------------------------------------------
// scalar slots in the device array S
// --------------------------------------------------------------------------
enum {
    S_RA = 0, S_RV, S_XA, S_XV,   // IR residual / solution norms (squared, by block)
    S_NRM, S_INVNRM,              // ||r||, 1/||r|| of the IR residual
    S_RR0, S_RR,                  // inner residual norms^2 (initial, current)
    S_RHO, S_ALPHA, S_OMEGA, S_BETA,
    S_RZ, S_RZ0,
    // the convergence test of a step captured whole (qk_cond_init / qk_cond_next)
    S_SREF = 23, S_REL, S_REL0, S_CYC, S_PRN, S_PRN_LAST,
    S_COUNT = 32
};

enum FinOp {
    FIN_RESID = 0, FIN_BICG_INIT, FIN_BICG_ALPHA, FIN_BICG_OMEGA, FIN_BICG_RHO,
    FIN_CG_INIT, FIN_CG_ALPHA, FIN_CG_BETA
};

__global__ void qk_finalize(const double* part, long long nb, int nsum, double* S, int op, unsigned* status) {
    pdl_wait();
    // a quarter of the block's warps per sum (16 warps, up to 4 sums), added up in a fixed order
    __shared__ double sh[4][4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, q = wid >> 2, part_w = wid & 3;
    if (q < nsum) {
        double acc = 0.0;
        for (long long t = part_w * 32 + lane; t < nb; t += 128) acc += part[q * nb + t];
        acc = qWarpSum(acc);
        if (lane == 0) sh[q][part_w] = acc;
    }
    __syncthreads();
    double sums[4];
    for (int i = 0; i < 4; i++) sums[i] = (sh[i][0] + sh[i][1]) + (sh[i][2] + sh[i][3]);
    if (threadIdx.x != 0) return;
    switch (op) {
    case FIN_RESID: {
        S[S_RA] = sums[0]; S[S_RV] = sums[1]; S[S_XA] = sums[2]; S[S_XV] = sums[3];
        double nr = sqrt(sums[0] + sums[1]);
        if (!isfinite(nr)) { atomicOr(status, (unsigned)QMS_ST_NAN); nr = 0.0; }
        S[S_NRM] = nr;
        S[S_INVNRM] = nr > 0.0 ? 1.0 / nr : 0.0;
        break;
    }
    case FIN_BICG_INIT:
        S[S_RR0] = sums[0]; S[S_RR] = sums[0]; S[S_RHO] = sums[0];
        S[S_ALPHA] = 1.0; S[S_OMEGA] = 1.0; S[S_BETA] = 0.0;
        break;
    case FIN_BICG_ALPHA: {
        double rv = sums[0];
        if (rv == 0.0 || !isfinite(rv)) { atomicOr(status, (unsigned)QMS_ST_BREAKDOWN); S[S_ALPHA] = 0.0; }
        else S[S_ALPHA] = S[S_RHO] / rv;
        break;
    }
    case FIN_BICG_OMEGA: {
        double ts = sums[0], tt = sums[1];
        S[S_OMEGA] = (tt > 0.0 && isfinite(tt)) ? ts / tt : 0.0;
        break;
    }
    case FIN_BICG_RHO: {
        double rho_new = sums[0];
        double om = S[S_OMEGA];
        if (S[S_RHO] == 0.0 || om == 0.0) { atomicOr(status, (unsigned)QMS_ST_BREAKDOWN); S[S_BETA] = 0.0; }
        else S[S_BETA] = (rho_new / S[S_RHO]) * (S[S_ALPHA] / om);
        S[S_RHO] = rho_new;
        S[S_RR] = sums[1];
        break;
    }
    case FIN_CG_INIT:
        S[S_RZ] = sums[0]; S[S_RZ0] = sums[0]; S[S_RR0] = sums[1]; S[S_RR] = sums[1];
        break;
    case FIN_CG_ALPHA: {
        double pq = sums[0];
        if (pq <= 0.0 || !isfinite(pq)) { atomicOr(status, (unsigned)QMS_ST_BREAKDOWN); S[S_ALPHA] = 0.0; }
        else S[S_ALPHA] = S[S_RZ] / pq;
        break;
    }
    case FIN_CG_BETA: {
        double rz_new = sums[0];
        S[S_BETA] = S[S_RZ] != 0.0 ? rz_new / S[S_RZ] : 0.0;
        S[S_RZ] = rz_new;
        S[S_RR] = sums[1];
        break;
    }
    }
}

// --------------------------------------------------------------------------
// convergence test of a whole step captured in one graph: the host loop's relative residual
// rel = |r| / min(max(|x|, s), 100 s), s = |x| at the start of the solve, from the finalized
// residual sums; the WHILE node runs another refinement cycle while rel > tol, at most
// maxcyc cycles, and while each cycle at least removes a tenth of the residual
// --------------------------------------------------------------------------
__global__ void qk_cond_init(double* __restrict__ S, double tol, cudaGraphConditionalHandle hc) {
    if (threadIdx.x != 0) return;
    const double xn = sqrt(S[S_XA] + S[S_XV]), rn = S[S_NRM];
    const double sref = xn > 0.0 ? xn : 1.0;
    const double rel = rn / fmin(fmax(xn, sref), 100.0 * sref);
    S[S_SREF] = sref;
    S[S_REL] = rel;
    S[S_REL0] = rel;
    S[S_CYC] = 0.0;
    S[S_PRN] = rn;
    S[S_PRN_LAST] = rn;
    cudaGraphSetConditional(hc, (isfinite(rel) && rel > tol && rn != 0.0) ? 1u : 0u);
}

__global__ void qk_cond_next(double* __restrict__ S, double tol, int maxcyc, cudaGraphConditionalHandle hc) {
    if (threadIdx.x != 0) return;
    const double xn = sqrt(S[S_XA] + S[S_XV]), rn = S[S_NRM], sref = S[S_SREF];
    const double rel = rn / fmin(fmax(xn, sref), 100.0 * sref);
    const double prev = S[S_PRN];
    const double cyc = S[S_CYC] + 1.0;
    S[S_CYC] = cyc;
    S[S_REL] = rel;
    S[S_PRN_LAST] = prev;
    S[S_PRN] = rn;
    const bool more = isfinite(rel) && rel > tol && rn != 0.0 && cyc < (double)maxcyc && rn < 0.9 * prev;
    cudaGraphSetConditional(hc, more ? 1u : 0u);
}

// --------------------------------------------------------------------------
// fused vector kernels (grid-stride; block partials for the dot products)
// --------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void store_partials(double* part, float a, float b) {
    __shared__ double sh[32];
    double s0 = qBlockSum(a, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s0;
    double s1 = qBlockSum(b, sh);
    if (threadIdx.x == 0) part[gridDim.x + blockIdx.x] = s1;
}

// r holds the normalised residual (converted from the FP64 residual): rh = r, p = v = e = 0
template <typename T>
__global__ void qk_bicg_init(long long n, const T* __restrict__ r, T* __restrict__ rh, T* __restrict__ p,
                             T* __restrict__ v, T* __restrict__ e, double* __restrict__ part) {
    float acc = 0.f;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const T rv = r[t];
        rh[t] = rv; p[t] = T(0); v[t] = T(0); e[t] = T(0);
        acc += (float)(rv * rv);
    }
    store_partials<T>(part, acc, 0.f);
}

template <typename T>
__global__ void qk_bicg_p(long long n, const T* __restrict__ r, T* __restrict__ p, const T* __restrict__ v,
                          const double* __restrict__ S) {
    const T beta = (T)S[S_BETA], om = (T)S[S_OMEGA];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        p[t] = r[t] + beta * (p[t] - om * v[t]);
}

template <typename T>
__global__ void qk_bicg_s(long long n, const T* __restrict__ r, const T* __restrict__ v, T* __restrict__ s,
                          const double* __restrict__ S) {
    const T al = (T)S[S_ALPHA];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        s[t] = r[t] - al * v[t];
}

template <typename T>
__global__ void qk_bicg_xr(long long n, const T* __restrict__ y, const T* __restrict__ z, const T* __restrict__ s,
                           const T* __restrict__ tt, const T* __restrict__ rh, T* __restrict__ e, T* __restrict__ r,
                           const double* __restrict__ S, double* __restrict__ part) {
    const T al = (T)S[S_ALPHA], om = (T)S[S_OMEGA];
    float a0 = 0.f, a1 = 0.f;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        T st = s[t];
        e[t] += al * y[t] + om * z[t];
        T rn = st - om * tt[t];
        r[t] = rn;
        a0 += (float)(rh[t] * rn);
        a1 += (float)(rn * rn);
    }
    store_partials<T>(part, a0, a1);
}

// r = D r, the unscaled residual of the normalised system (r holds the normalised scaled
// residual converted from the FP64 one), e = 0
template <typename T>
__global__ void qk_cg_init(long long n, const float* __restrict__ dg, T* __restrict__ r, T* __restrict__ e) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        r[t] = (T)dg[t] * r[t];
        e[t] = T(0);
    }
}

// Jacobi preconditioner of the unscaled system (V block frozen when mask_from < n)
template <typename T>
__global__ void qk_jacobi(long long n, long long mask_from, const T* __restrict__ r, const float* __restrict__ dg,
                          T* __restrict__ z) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const float d = dg[t];                   // 0 on the padding of the layout
        z[t] = t < mask_from && d != 0.f ? r[t] / (T)d : T(0);
    }
}

// 16-byte packets: the padded layout's length is a multiple of 4 elements and every vector
// starts on a 256-byte boundary, so sweeps over vectors move whole packets
template <typename T> struct GmPack;
template <> struct GmPack<float> {
    using V = float4;
    static constexpr int W = 4;
    static __device__ __forceinline__ float at(const V& v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }
};
template <> struct GmPack<double> {
    using V = double2;
    static constexpr int W = 2;
    static __device__ __forceinline__ double at(const V& v, int q) { return q == 0 ? v.x : v.y; }
};

// the products of two packets, added up in T: a thread's FP32 sum then takes one number per packet
template <typename T>
__device__ __forceinline__ float gm_dot(const typename GmPack<T>::V& a, const typename GmPack<T>::V& b) {
    T s = GmPack<T>::at(a, 0) * GmPack<T>::at(b, 0);
#pragma unroll
    for (int q = 1; q < GmPack<T>::W; q++) s += GmPack<T>::at(a, q) * GmPack<T>::at(b, q);
    return (float)s;
}

// The conjugate-gradient vectors, 16-byte packets over the three A blocks (the V block is frozen at
// zero).  Bound by bytes: e takes its step together with p's (one read of p less than apart), 9 blocks
// of vector traffic per iteration in all where 13 were (V block included).
template <typename T>
__device__ __forceinline__ long long cg_packets(long long n) { return n * (long long)sizeof(T) / 16; }

// partials of r.z and z.z; optionally p = z (first iteration)
template <typename T>
__global__ void __launch_bounds__(256) qk_cg_dot(long long n, const T* r, const T* z, T* p, double* part) {
    using PK = GmPack<T>;
    using PV = typename PK::V;
    float a0 = 0.f, a1 = 0.f;
    pdl_wait();
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < cg_packets<T>(n); t += (long long)gridDim.x * blockDim.x) {
        const PV zv = reinterpret_cast<const PV*>(z)[t], rv = reinterpret_cast<const PV*>(r)[t];
        if (p) reinterpret_cast<PV*>(p)[t] = zv;
#pragma unroll
        for (int q = 0; q < PK::W; q++) {
            a0 += (float)(PK::at(rv, q) * PK::at(zv, q));
            a1 += (float)(PK::at(zv, q) * PK::at(zv, q));
        }
    }
    store_partials<T>(part, a0, a1);
}

// v += sign alpha d
template <typename T>
__global__ void __launch_bounds__(256) qk_cg_axpy(long long n, const T* d, const double* S, T sign, T* v) {
    using PK = GmPack<T>;
    using PV = typename PK::V;
    pdl_wait();
    const T al = sign * (T)S[S_ALPHA];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < cg_packets<T>(n); t += (long long)gridDim.x * blockDim.x) {
        const PV dv = reinterpret_cast<const PV*>(d)[t];
        PV vv = reinterpret_cast<PV*>(v)[t];
        T* vq = reinterpret_cast<T*>(&vv);
#pragma unroll
        for (int q = 0; q < PK::W; q++) vq[q] += al * PK::at(dv, q);
        reinterpret_cast<PV*>(v)[t] = vv;
    }
}

// e += alpha p, then p = z + beta p
template <typename T>
__global__ void __launch_bounds__(256) qk_cg_ep(long long n, const T* z, T* p, T* e, const double* S) {
    using PK = GmPack<T>;
    using PV = typename PK::V;
    pdl_wait();
    const T al = (T)S[S_ALPHA], be = (T)S[S_BETA];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < cg_packets<T>(n); t += (long long)gridDim.x * blockDim.x) {
        const PV zv = reinterpret_cast<const PV*>(z)[t];
        PV pv = reinterpret_cast<PV*>(p)[t], ev = reinterpret_cast<PV*>(e)[t];
        T* pq = reinterpret_cast<T*>(&pv);
        T* eq = reinterpret_cast<T*>(&ev);
#pragma unroll
        for (int q = 0; q < PK::W; q++) {
            eq[q] += al * pq[q];
            pq[q] = PK::at(zv, q) + be * pq[q];
        }
        reinterpret_cast<PV*>(p)[t] = pv;
        reinterpret_cast<PV*>(e)[t] = ev;
    }
}

// --------------------------------------------------------------------------
// FGMRES (right preconditioned, restarted by the outer refinement) with the
// Hessenberg matrix, Givens rotations and the residual estimate on the device.
// --------------------------------------------------------------------------
// basis of up to 64 vectors; the Gram-Schmidt and update kernels take at most GM_PASS of them
// per launch (compile-time counts), so longer bases run as two passes
#define GM_MAXM 64
#define GM_PASS 32
struct GmPtrs { const void* p[GM_MAXM + 1]; };

// True in every thread of the block that arrives last (its threads then see what the others wrote
// before); the counter is zero again for the next launch.
__device__ __forceinline__ bool gm_last_block(unsigned* counter) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
        if (last) *counter = 0;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Classical Gram-Schmidt projections.  NV is a compile-time count so every load of the unrolled loop is
// unconditional and independent (memory-level parallelism over all basis vectors).
// h_ij = V_i . w for i < NV, and w . w, as block partials (row i of `part`, rows of gridDim.x); in
// the last pass over the basis (final) the last block adds them up in a fixed order into column j
// of H and forms the norm of the orthogonalised w from Pythagoras, |w'|^2 = |w|^2 - sum_i h_ij^2:
// when that keeps at least a hundredth of |w|^2 (no severe cancellation), Gm[4] = |w'| and Gm[3]
// = 1, and the orthogonalisation writes V_{j+1} = w' / |w'| directly (no norm pass over w', no
// scaling pass); otherwise Gm[3] = 0.  row0: the basis vectors of the passes before; part0: row 0.
// On large grids the basis vectors' bandwidth bounds this (256^3: 85-90 % of the copy rate); on
// small ones the tail did: a block sum with two barriers per vector and a one-block kernel that
// added up one vector after the other.  Now the warps leave their sums in shared memory behind one
// barrier, and each warp of the last block adds up vectors of its own (48^3: 240 ms per run of 8
// steps instead of 299, 64x64x80 core 261 instead of 303).  The grid is one resident wave: with
// eight blocks per SM whatever the registers, a second wave of a few blocks followed (256^3, 8
// vectors: 367 us instead of 405).
// A thread then adds up more, one number per packet (gm_dot): at 256^3 w . w is 0.6e-9 to 1.1e-9 of itself
// off with six and three blocks per SM, 1.8e-9 to 8.5e-9 with an addition per element, and was 1.4e-9 with
// eight blocks (normal random w); V_i . w is 0.7e-11 to 1.8e-11 of |V_i| |w| off, and was 5.0e-11.
template <typename T, int NV>
__global__ void __launch_bounds__(256) qk_gm_dots(long long n, GmPtrs V, const T* w, double* part0, int row0,
                                                  int final, int j, int m, double* Hm, double* Gm,
                                                  unsigned* counter) {
    using PK = GmPack<T>;
    using PV = typename PK::V;
    float acc[NV + 1];
#pragma unroll
    for (int i = 0; i <= NV; i++) acc[i] = 0.f;
    const PV* vp[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) vp[i] = (const PV*)V.p[i];
    const PV* wp = (const PV*)w;
    const long long np = n / PK::W;
    pdl_wait();
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < np; t += (long long)gridDim.x * blockDim.x) {
        const PV wv = wp[t];
        PV vv[NV];
#pragma unroll
        for (int i = 0; i < NV; i++) vv[i] = __ldg(vp[i] + t);
#pragma unroll
        for (int i = 0; i < NV; i++) acc[i] += gm_dot<T>(vv[i], wv);
        acc[NV] += gm_dot<T>(wv, wv);
    }
    __shared__ double sums[GM_MAXM + 2];
    __shared__ float sh[NV + 1][8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i <= NV; i++) {
        const float s = qWarpSum(acc[i]);
        if (lane == 0) sh[i][wid] = s;
    }
    __syncthreads();
    if (threadIdx.x <= NV) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < 8; q++) s += (double)sh[threadIdx.x][q];
        part0[(long long)(row0 + threadIdx.x) * gridDim.x + blockIdx.x] = s;
    }
    if (!final || !gm_last_block(counter)) return;
    for (int i = wid; i <= j + 1; i += 8) {
        double s = 0.0;
        for (int t = lane; t < (int)gridDim.x; t += 32) s += __ldcg(part0 + (long long)i * gridDim.x + t);
        s = qWarpSum(s);
        if (lane == 0) sums[i] = s;
    }
    __syncthreads();
    if ((int)threadIdx.x <= j) Hm[threadIdx.x * m + j] = sums[threadIdx.x];
    if (threadIdx.x == 0) {
        double hh = 0.0;
        for (int i = 0; i <= j; i++) hh += sums[i] * sums[i];
        const double s = sums[j + 1], est = s - hh;
        const bool ok = isfinite(est) && est > 1e-2 * s;
        Gm[3] = ok ? 1.0 : 0.0;
        Gm[4] = ok ? sqrt(est) : 0.0;
    }
}

// w' = w - sum_i h_ij V_i (NV basis vectors, compile-time; 16-byte packets): with Gm[3] set, V_{j+1}
// = w' / Gm[4] goes to vout; otherwise w' back into w with the partials of |w'|^2.
// final = 0: a first pass over part of the basis (w' back into w, no norm partials, no direct write).
// In the last pass the last block (every block has read column j of H by then) takes h_{j+1,j} = |w'|,
// applies the Givens rotations and forms the residual estimate; Gm layout: [0]: beta,
// [1]: |g_{j+1}|, [2]: 1/h_{j+1,j}, cs[m] at 8, sn[m] at 8+m, g[m+1] at 8+2m
template <typename T, int NV>
__global__ void __launch_bounds__(256) qk_gm_orth(long long n, int j, int m, GmPtrs V, double* Hcol0, int row0,
                                                  T* w, double* part, double* Gm, T* vout, int final,
                                                  unsigned* counter, unsigned* status) {
    using PK = GmPack<T>;
    using PV = typename PK::V;
    T h[NV];
    const PV* vp[NV];
    pdl_wait();
#pragma unroll
    for (int i = 0; i < NV; i++) { h[i] = (T)Hcol0[(row0 + i) * m + j]; vp[i] = (const PV*)V.p[i]; }
    const bool direct = final && Gm[3] != 0.0;
    const T inv = direct ? (T)(1.0 / Gm[4]) : T(1);
    PV* wp = (PV*)w;
    PV* op = direct ? (PV*)vout : wp;
    const long long np = n / PK::W;
    float acc = 0.f;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < np; t += (long long)gridDim.x * blockDim.x) {
        PV vv[NV];
#pragma unroll
        for (int i = 0; i < NV; i++) vv[i] = __ldg(vp[i] + t);
        PV wv = wp[t];
        T* wq = reinterpret_cast<T*>(&wv);
#pragma unroll
        for (int q = 0; q < PK::W; q++) {
            T a = wq[q];
#pragma unroll
            for (int i = 0; i < NV; i++) a -= h[i] * PK::at(vv[i], q);
            wq[q] = direct ? a * inv : a;
            acc += (float)(a * a);
        }
        op[t] = wv;
    }
    if (!final) return;
    __shared__ double sh[32];
    if (!direct) {
        const double s0 = qBlockSum(acc, sh);
        if (threadIdx.x == 0) part[blockIdx.x] = s0;
    }
    if (!gm_last_block(counter)) return;
    double nw = 0.0;
    if (!direct) {
        for (int t = threadIdx.x; t < (int)gridDim.x; t += blockDim.x) nw += __ldcg(part + t);
        nw = qBlockSum(nw, sh);
    }
    // column j of H and the rotations in shared memory: the chain of rotations is one thread's
    __shared__ double hc[GM_MAXM + 1], rc[GM_MAXM], rs[GM_MAXM];
    if ((int)threadIdx.x <= j) hc[threadIdx.x] = __ldcg(Hcol0 + threadIdx.x * m + j);
    if ((int)threadIdx.x < j) {
        rc[threadIdx.x] = Gm[8 + threadIdx.x];
        rs[threadIdx.x] = Gm[8 + m + threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double hn = direct ? Gm[4] : sqrt(nw);
        double* gv = Gm + 8 + 2 * m;
        Gm[2] = hn > 0.0 ? 1.0 / hn : 0.0;
        double b = hc[0];
        for (int i = 0; i < j; i++) {                // previous rotations on column j
            const double a = b, c = hc[i + 1];
            hc[i] = rc[i] * a + rs[i] * c;
            b = -rs[i] * a + rc[i] * c;
        }
        const double r = sqrt(b * b + hn * hn);
        const double c = r > 0.0 ? b / r : 1.0, s = r > 0.0 ? hn / r : 0.0;
        Gm[8 + j] = c;
        Gm[8 + m + j] = s;
        hc[j] = r;
        const double gj = gv[j];
        gv[j + 1] = -s * gj;
        gv[j] = c * gj;
        Gm[1] = fabs(s * gj);
        if (!(r > 0.0) || !isfinite(r)) atomicOr(status, (unsigned)QMS_ST_BREAKDOWN);
    }
    __syncthreads();
    if ((int)threadIdx.x <= j) Hcol0[threadIdx.x * m + j] = hc[threadIdx.x];
}

// V_{j+1} = w / h_{j+1,j} (nothing to do when the orthogonalisation wrote it, Gm[3])
template <typename T>
__global__ void qk_gm_scale(long long n, const T* w, T* vout, const double* Gm) {
    pdl_wait();
    if (Gm[3] != 0.0) return;
    const T inv = (T)Gm[2];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        vout[t] = w[t] * inv;
}


__global__ void qk_gm_reset(int m, double* __restrict__ Gm) {
    for (int q = threadIdx.x; q < 8 + 3 * m + 1; q += blockDim.x) Gm[q] = 0.0;
    __syncthreads();
    if (threadIdx.x == 0) { Gm[0] = 1.0; Gm[8 + 2 * m] = 1.0; Gm[1] = 1.0; }
}

// back substitution H(0:k,0:k) y = g(0:k), column by column in one warp (lane l holds the right-hand
// sides of rows l and l + 32); y stored at Gm + 8 + 3m + 1
__global__ void __launch_bounds__(256) qk_gm_solve(int k, int m, const double* __restrict__ Hm,
                                                  double* __restrict__ Gm) {
    __shared__ double hs[GM_MAXM * GM_MAXM];
    for (int q = threadIdx.x; q < k * k; q += blockDim.x) hs[q] = Hm[(q / k) * m + q % k];
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const double* gv = Gm + 8 + 2 * m;
    double* y = Gm + 8 + 3 * m + 1;
    double a0 = lane < k ? gv[lane] : 0.0, a1 = lane + 32 < k ? gv[lane + 32] : 0.0;
    for (int i = k - 1; i >= 0; i--) {
        const double d = hs[i * k + i];
        const double acc = __shfl_sync(0xffffffffu, i >= 32 ? a1 : a0, i & 31);
        const double yi = d != 0.0 ? acc / d : 0.0;
        if (lane == 0) y[i] = yi;
        if (lane < i) a0 -= hs[lane * k + i] * yi;
        if (lane + 32 < i) a1 -= hs[(lane + 32) * k + i] * yi;
    }
}

// x[ref] += nrm * sum_i y_i Z_i[PL]   (FP64 accumulation of the refinement); one thread per
// node, its (up to) four unknowns
template <typename T, int NV>
__global__ void __launch_bounds__(QMS_NODE_BX * QMS_NODE_BY) qk_gm_update(QGrid g, int m, GmPtrs Z, const double* __restrict__ Gm,
                                                    const double* __restrict__ S, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z + 1;
    if (i > g.Nx || j > g.Ny) return;
    const double* yv = Gm + 8 + 3 * m + 1;
    T y[NV];
    const T* zp[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) { y[q] = (T)yv[q]; zp[q] = (const T*)Z.p[q]; }
    const double nr = S[S_NRM];
    const QPL L = qms_pl(g);
    const long long nd = qms_pl_node(g, L, i, j, k);
    auto comb = [&](long long t) {
        T acc = T(0);
#pragma unroll
        for (int q = 0; q < NV; q++) acc += y[q] * __ldg(zp[q] + t);
        return nr * (double)acc;
    };
    if (i <= g.xs) x[qAX(g, i, j, k)] += comb(nd);
    if (j <= g.ys) x[qAY(g, i, j, k)] += comb(L.comp + nd);
    if (k <= g.zs) x[qAZ(g, i, j, k)] += comb(2 * L.comp + nd);
    x[qV(g, i, j, k)] += comb(3 * L.comp + nd);
}

// compile-time dispatch on the number of basis vectors (1..GM_MAXM)
#define GM_CASES(M) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13) M(14) M(15) M(16) \
    M(17) M(18) M(19) M(20) M(21) M(22) M(23) M(24) M(25) M(26) M(27) M(28) M(29) M(30) M(31) M(32)

static GmPtrs gm_shift(const GmPtrs& V, int off) {
    GmPtrs r{};
    for (int i = 0; i + off <= GM_MAXM; i++) r.p[i] = V.p[i + off];
    return r;
}
// One resident wave of blocks (at most vb): each walks the vectors with the same stride, so blocks of a
// second, partial wave would run while most SMs have nothing left
static int gm_blocks(const void* kernel, std::atomic<int>& per, int vb, int nsm) {
    int p = per.load(std::memory_order_relaxed);
    if (p == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, kernel, 256, 0);
        p = std::max(1, p);
        per.store(p, std::memory_order_relaxed);
    }
    return std::min(vb, nsm * p);
}
// return the kernel launches
template <typename T>
static int gm_dots(int nv, int vb, cudaStream_t st, long long n, const GmPtrs& V, const T* w, double* part, int row0,
                   int j, int m, double* Hm, double* Gm, unsigned* counter, int nsm) {
    const int now = std::min(nv, GM_PASS), final = now == nv ? 1 : 0;
    int nb = vb;                                // later passes: as many blocks (partials) as the first
    switch (now) {
#define C(N) case N: { static std::atomic<int> per{0}; \
        if (row0 == 0) nb = gm_blocks((const void*)qk_gm_dots<T, N>, per, vb, nsm); \
        pdl_launch(qk_gm_dots<T, N>, dim3(nb), dim3(256), 0, st, 0, n, V, w, part, row0, final, j, m, Hm, Gm, counter); } break;
        GM_CASES(C)
#undef C
    }
    return final ? 1 : 1 + gm_dots<T>(nv - now, nb, st, n, gm_shift(V, now), w, part, row0 + now, j, m, Hm, Gm, counter, nsm);
}
template <typename T>
static int gm_orth(int nv, int vb, cudaStream_t st, long long n, int j, int m, const GmPtrs& V, double* Hm, int row0,
                   T* w, double* part, double* Gm, T* vout, unsigned* counter, unsigned* status, int nsm) {
    const int now = std::min(nv, GM_PASS), final = now == nv ? 1 : 0;
    switch (now) {
#define C(N) case N: { static std::atomic<int> per{0}; \
        pdl_launch(qk_gm_orth<T, N>, dim3(gm_blocks((const void*)qk_gm_orth<T, N>, per, vb, nsm)), dim3(256), 0, st, 0, n, j, m, V, Hm, row0, w, part, Gm, vout, final, counter, status); } break;
        GM_CASES(C)
#undef C
    }
    return final ? 1 : 1 + gm_orth<T>(nv - now, vb, st, n, j, m, gm_shift(V, now), Hm, row0 + now, w, part, Gm, vout,
                                      counter, status, nsm);
}
template <typename T>
static int gm_update(int nv, cudaStream_t st, const QGrid& g, int m, const GmPtrs& Z, const double* Gm,
                     const double* S, double* x) {
    if (nv > GM_PASS) {
        // x += nr (sum of the first GM_PASS terms) + nr (the rest): the y of the second pass start
        // GM_PASS further into Gm
        gm_update<T>(GM_PASS, st, g, m, Z, Gm, S, x);
        return 1 + gm_update<T>(nv - GM_PASS, st, g, m, gm_shift(Z, GM_PASS), Gm + GM_PASS, S, x);
    }
    switch (nv) {
#define C(N) case N: qk_gm_update<T, N><<<qms_node_grid(g), qms_node_block(), 0, st>>>(g, m, Z, Gm, S, x); break;
        GM_CASES(C)
#undef C
    }
    return 1;
}


// --------------------------------------------------------------------------
// material table
// --------------------------------------------------------------------------
template <typename T>
void qms_fill_table(QMatTable<T>& t, const double* rows6, int nmat) {
    for (int s = 0; s < QMS_MAX_SLOTS; s++) {
        for (int d = 0; d < 3; d++) {
            double mu = QMS_MU0, sg = 0.0;                    // slot 0 and unused slots: vacuum (F:211-225)
            if (s >= 1 && s <= nmat) {
                mu = rows6[(s - 1) * 6 + d] * QMS_MU0;        // F:245-247
                sg = rows6[(s - 1) * 6 + 3 + d];              // F:248-250
            }
            t.mu[3 * s + d] = (T)mu;
            t.imu[3 * s + d] = (T)(1.0 / mu);
            t.sig[3 * s + d] = (T)sg;
        }
    }
}
template void qms_fill_table<double>(QMatTable<double>&, const double*, int);
template void qms_fill_table<float>(QMatTable<float>&, const double*, int);

// --------------------------------------------------------------------------
// solver object
// --------------------------------------------------------------------------
#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t _e = (call);                                                          \
        if (_e != cudaSuccess) {                                                          \
            err = std::string(#call) + ": " + cudaGetErrorString(_e);                     \
            return QMS_ERR_CUDA;                                                          \
        }                                                                                 \
    } while (0)

QmsSolver::~QmsSolver() { release(); }

void QmsSolver::release() {
    if (dev >= 0) cudaSetDevice(dev);
    mgf[0].release(); mgf[1].release(); mgd[0].release(); mgd[1].release();
    for (auto& p : gmV) { if (p) cudaFree(p); p = nullptr; }
    for (auto& p : gmZ) { if (p) cudaFree(p); p = nullptr; }
    if (gm_H) cudaFree(gm_H);
    if (gm_scal) cudaFree(gm_scal);
    if (gm_count) cudaFree(gm_count);
    gm_H = gm_scal = nullptr;
    gm_count = nullptr;
    if (nc16) cudaFree(nc16);
    nc16 = nullptr;
    void* ptrs[] = {ids,   dtab64, dtab32,    x,     b,      r64,    xbest, H,   slicebuf, part,   S,
                    status, dg_steady, dg_tr, mgtmp, mgtmp2, nc32,  nc64,  xdf, r0df,     ncdf, rpl, x0,
                    rsg,   rsdt,   bprev,     rfin,  dinvdf, xold, xold2, hist_x, xold3, wh[0], wh[1], wh[2],
                    wh[3], xold4, lsp, lsg};
    for (void* q : ptrs) if (q) cudaFree(q);
    if (hS) cudaFreeHost(hS);
    if (hptrs) cudaFreeHost(hptrs);
    if (dptrs) cudaFree(dptrs);
    hptrs = nullptr;
    dptrs = nullptr;
    for (auto& p : vec) if (p) cudaFree(p);
    drop_graphs();
    for (auto& e : evpool) { cudaEventDestroy(e.a); cudaEventDestroy(e.b); }
    evpool.clear();
    for (int q = 0; q < kFieldSlots; q++) {
        if (fev_done[q]) cudaEventSynchronize(fev_done[q]);
        if (fev_ready[q]) cudaEventDestroy(fev_ready[q]);
        if (fev_done[q]) cudaEventDestroy(fev_done[q]);
        if (fbuf[q]) cudaFree(fbuf[q]);
        fev_ready[q] = fev_done[q] = nullptr;
        fbuf[q] = nullptr;
        fbuf_n[q] = 0;
    }
    if (cst) cudaStreamDestroy(cst);
    cst = nullptr;
    if (st && own_stream) cudaStreamDestroy(st);
    ids = nullptr; dtab64 = nullptr; dtab32 = nullptr; x = b = r64 = H = slicebuf = part = S = nullptr;
    status = nullptr; dg_steady = dg_tr = nullptr; hS = nullptr; st = nullptr; mgtmp = nullptr; mgtmp2 = nullptr; xbest = nullptr;
    xdf = r0df = ncdf = nullptr; rpl = nullptr; x0 = nullptr; df_resid = false; anchor_ready = false;
    rsg = rsdt = nullptr;
    bprev = nullptr; rfin = dinvdf = nullptr; rfin_ok = false; chain_len = 0; xold = xold2 = nullptr;
    hist_x = nullptr; hist_len = 0; xold3 = xold4 = nullptr; wh[0] = wh[1] = wh[2] = wh[3] = nullptr; w_len = 0;
    nwh = 0; lsp = lsg = nullptr; last_chained = false;
    field_run = 0; start_resid_ready = false;
    nc32 = nullptr; nc64 = nullptr;
    for (auto& p : vec) p = nullptr;
}

int QmsSolver::init(const qms_desc& d) {
    desc = d;
    mghook.s = this;
    for (int q = 0; q < 2; q++) { mgf[q].prof = &mghook; mgd[q].prof = &mghook; }
    dev = d.device;
    CK(cudaSetDevice(dev));
    if (d.xs < 4 || d.ys < 4 || d.zs < 4) { err = "grid must have at least 4 cells per axis"; return QMS_ERR_ARG; }
    if (!(d.dx > 0 && d.dy > 0 && d.dz > 0 && d.dt > 0)) { err = "dx, dy, dz, dt must be positive"; return QMS_ERR_ARG; }
    g = qms_make_grid(d.xs, d.ys, d.zs, d.dx, d.dy, d.dz);
    // the stencil kernels index rows with 32-bit integers (and the padded layout is a little larger)
    npl = qms_pl(g).n;
    if (g.n >= 0x7fffffffLL || npl >= 0x7fffffffLL) {
        err = "grid too large: more than 2^31 - 1 unknowns";
        return QMS_ERR_ARG;
    }
    fp64_inner = d.precision == QMS_PREC_FP64;
    trace = std::getenv("QMS_TRACE") != nullptr;
    tsize = fp64_inner ? sizeof(double) : sizeof(float);
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    vec_blocks = (long long)nsm * 8;
    long long need = (npl + 255) / 256;
    if (need < vec_blocks) vec_blocks = need;
    nbop = qms_op_num_blocks(g);
    nbpl = qms_op_pl_num_blocks(g);
    long long npart = std::max(4 * std::max(nbop, nbpl), (long long)(GM_MAXM + 1) * vec_blocks) + 64;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    own_stream = true;
    const long long n = g.n, ncell = (long long)g.xs * g.ys * g.zs;
    CK(cudaMalloc(&ids, ncell));
    CK(cudaMemsetAsync(ids, 0, ncell, st));
    CK(cudaMalloc(&dtab64, sizeof(QMatTable<double>)));
    CK(cudaMalloc(&dtab32, sizeof(QMatTable<float>)));
    CK(cudaMalloc(&x, n * 8));
    CK(cudaMalloc(&b, n * 8));
    CK(cudaMalloc(&r64, n * 8));
    CK(cudaMalloc(&xbest, n * 8));
    CK(cudaMalloc(&H, 3 * ncell * 8));
    long long smax = std::max({(long long)g.ys * g.zs, (long long)g.xs * g.zs, (long long)g.xs * g.ys});
    CK(cudaMalloc(&slicebuf, 3 * smax * 8));
    CK(cudaMalloc(&part, npart * 8));
    CK(cudaMalloc(&S, S_COUNT * 8));
    CK(cudaMemsetAsync(S, 0, S_COUNT * 8, st));
    CK(cudaMalloc(&status, sizeof(unsigned)));
    CK(cudaMemsetAsync(status, 0, sizeof(unsigned), st));
    CK(cudaMalloc(&nc32, 6 * qms_pl(g).comp * 4));
    CK(cudaMalloc(&nc64, 6 * qms_pl(g).comp * 8));
    // inner-solver vectors in the padded layout; the padding stays zero
    auto pl_alloc = [&](void** p, size_t es) -> cudaError_t {
        cudaError_t e = cudaMalloc(p, npl * es);
        return e != cudaSuccess ? e : cudaMemsetAsync(*p, 0, npl * es, st);
    };
    CK(pl_alloc((void**)&dg_steady, 4));
    CK(pl_alloc((void**)&dg_tr, 4));
    for (auto& p : vec) CK(pl_alloc(&p, tsize));
    // multigrid needs at least two levels (grids of a few cells use the Jacobi / identity fallback)
    use_mg = d.precond == QMS_PRECOND_MG && QmsMG<float>::levels_for(g, 5) >= 2;
    CK(pl_alloc((void**)&mgtmp, tsize));
    if (use_mg) CK(pl_alloc((void**)&mgtmp2, tsize));
    if (d.krylov == QMS_KRYLOV_GMRES) {
        const int m = std::min(std::max(d.gmres_m, 1), GM_MAXM);
        desc.gmres_m = m;
        for (int i = 0; i <= m; i++) CK(pl_alloc(&gmV[i], tsize));
        if (use_mg) for (int i = 0; i < m; i++) CK(pl_alloc(&gmZ[i], tsize));
        CK(cudaMalloc(&gm_H, (size_t)m * (m + 1) * 8));
        CK(cudaMalloc(&gm_scal, (size_t)(8 + 4 * m + 8) * 8));
        CK(cudaMalloc(&gm_count, sizeof(unsigned)));
        CK(cudaMemsetAsync(gm_count, 0, sizeof(unsigned), st));
    }
    CK(cudaMallocHost(&hS, S_COUNT * 8));
    CK(cudaMemsetAsync(x, 0, n * 8, st));
    // tensor maps of every padded vector that feeds a stencil kernel, and of the coefficients
    std::vector<const void*> mapped(vec, vec + QMS_NVEC);
    mapped.push_back(mgtmp);
    for (int i = 0; i <= GM_MAXM; i++) if (gmV[i]) mapped.push_back(gmV[i]);
    for (int i = 0; i < GM_MAXM; i++) if (gmZ[i]) mapped.push_back(gmZ[i]);
    if (mgtmp2) mapped.push_back(mgtmp2);
    if (!fp64_inner) {
        df_resid = true;
        CK(pl_alloc((void**)&xdf, 8));
        CK(pl_alloc((void**)&r0df, 8));
        CK(cudaMalloc(&rsg, g.oV * 8));
        CK(cudaMalloc(&rsdt, g.oV * 8));
        CK(cudaMalloc(&bprev, n * 8));
        CK(cudaMalloc(&xold, n * 8));
        CK(cudaMalloc(&hist_x, n * 8));
        const int hx_need = std::max(std::min(d.extrapolate, 3), d.start_ls);   // history beyond x_n, x_(n-1)
        if (hx_need >= 2) CK(cudaMalloc(&xold2, n * 8));
        if (hx_need >= 3) CK(cudaMalloc(&xold3, n * 8));
        if (hx_need >= 4) CK(cudaMalloc(&xold4, n * 8));
        nwh = hx_need;
        for (int q = 0; q < nwh; q++) CK(pl_alloc((void**)&wh[q], 8));
        if (d.start_ls > 0) {
            CK(cudaMalloc(&lsp, (size_t)QMS_LS_SUMS * nbpl * 8));
            CK(cudaMalloc(&lsg, 8 * 8));
        }
        CK(pl_alloc((void**)&rfin, 8));
        CK(pl_alloc((void**)&dinvdf, 8));
        CK(cudaMalloc(&x0, n * 8));
        CK(pl_alloc((void**)&rpl, 4));
        CK(cudaMallocHost(&hptrs, sizeof(QStepPtrs)));
        CK(cudaMalloc(&dptrs, sizeof(QStepPtrs)));
        CK(cudaMalloc(&ncdf, 6 * qms_pl(g).comp * 8));
        CK(cudaMemsetAsync(ncdf, 0, 6 * qms_pl(g).comp * 8, st));
        if (!qms_make_pl_map(&xdfmap, xdf, g, 8, 4, PLXY) || !qms_make_pl_map(&cdfmap, ncdf, g, 8, 6, PLCY)) {
            err = "tensor map encoding failed";
            return QMS_ERR_CUDA;
        }
    }
    const long long vbytes = 3 * qms_pl(g).comp * (long long)tsize;   // offset of the V block
    for (const void* p : mapped) {
        CUtensorMap mp, ma, mv;
        if (!qms_make_pl_map(&mp, p, g, (int)tsize, 4, PLXY) || !qms_make_pl_map(&ma, p, g, (int)tsize, 3, PLXY) ||
            !qms_make_pl_map(&mv, (const char*)p + vbytes, g, (int)tsize, 1, PLXY)) {
            err = "tensor map encoding failed";
            return QMS_ERR_CUDA;
        }
        tmaps[p] = mp;
        tmapsA[p] = ma;
        tmapsV[p] = mv;
    }
    if (!fp64_inner) {
        const long long comp16 = (long long)qms_pl16_pitch(g) * g.Ny * g.Nz;
        CK(cudaMalloc(&nc16, 6 * comp16 * sizeof(__nv_bfloat16)));
        if (!qms_make_pl16_map(&cmap16, nc16, g, 6) || !qms_make_pl16_map(&cmapV16, nc16 + 3 * comp16, g, 3)) {
            err = "tensor map encoding failed";
            return QMS_ERR_CUDA;
        }
    }
    const long long cv = 3 * qms_pl(g).comp;                          // first conductivity array
    if (!qms_make_pl_map(&cmap32, nc32, g, 4, 6, PLCY) || !qms_make_pl_map(&cmap64, nc64, g, 8, 6, PLCY) ||
        !qms_make_pl_map(&cmapV32, nc32 + cv, g, 4, 3, PLCY) || !qms_make_pl_map(&cmapV64, nc64 + cv, g, 8, 3, PLCY)) {
        err = "tensor map encoding failed";
        return QMS_ERR_CUDA;
    }
    double vac[6] = {1, 1, 1, 0, 0, 0};
    return set_materials(nullptr, vac, 0);
}

size_t qms_device_bytes_impl(const qms_desc& d) {
    QGrid g = qms_make_grid(d.xs, d.ys, d.zs, d.dx, d.dy, d.dz);
    size_t ts = d.precision == QMS_PREC_FP64 ? 8 : 4;
    // the block-triangular preconditioner's V right-hand side; the double-float residual's x, b,
    // coefficients and FP32 result (mixed precision)
    size_t tri = d.precond == QMS_PRECOND_MG ? qms_pl(g).n * ts : 0;
    // history of the extrapolated and least-squares starts: x_(n-2).. and the residual images
    const int lsn = std::max(0, std::min(d.start_ls, 4));
    const size_t hxn = (size_t)std::max(std::max(0, std::min(d.extrapolate, 3)), lsn);
    if (ts == 4) tri += (size_t)6 * qms_pl16_pitch(g) * g.Ny * g.Nz * 2;       // bf16 node coefficients
    if (ts == 4) tri += qms_pl(g).n * (8 + 8 + 4 + 8 + 8) + 6 * qms_pl(g).comp * 8 + 5 * g.n * 8 + 2 * g.oV * 8 +
                        (hxn > 2 ? hxn - 2 : 0) * g.n * 8 + hxn * qms_pl(g).n * 8 +
                        (lsn > 0 ? (QMS_LS_SUMS * (size_t)qms_op_pl_num_blocks(g) + 8) * 8 : 0);
    size_t ncell = (size_t)g.xs * g.ys * g.zs;
    size_t smax = std::max({(size_t)g.ys * g.zs, (size_t)g.xs * g.zs, (size_t)g.xs * g.ys});
    size_t nb = (size_t)std::max(qms_op_num_blocks(g), qms_op_pl_num_blocks(g));
    return tri + ncell + sizeof(QMatTable<double>) + sizeof(QMatTable<float>) + 4 * g.n * 8 + 3 * ncell * 8 +
           6 * qms_pl(g).comp * 12 +
           3 * smax * 8 + (4 * nb + 64) * 8 + 2 * qms_pl(g).n * 4 + (QMS_NVEC + 1) * qms_pl(g).n * ts + 4096 +
           (d.krylov == QMS_KRYLOV_GMRES ? (size_t)(2 * d.gmres_m + 1) * qms_pl(g).n * ts : 0) +
           (d.precond == QMS_PRECOND_MG ? 2 * (ts == 8 ? QmsMG<double>::bytes_for(g, 5, true) : QmsMG<float>::bytes_for(g, 5, true)) : 0) +
           // conductor-region coarse space: node lists (at most every node) and the K x K pseudo-inverse
           (d.precond == QMS_PRECOND_MG ? (size_t)g.Nn * 8 + (size_t)QMS_REGION_MAX * QMS_REGION_MAX * 8 + 64 * 1024 : 0);
}

int QmsSolver::set_materials(const uint8_t* host_slots, const double* rows6, int nmat) {
    CK(cudaSetDevice(dev));
    drop_graphs();
    forget_counts();
    if (nmat < 0 || nmat > QMS_MAX_SLOTS - 1) { err = "nmat must be in 0..255"; return QMS_ERR_ARG; }
    const long long ncell = (long long)g.xs * g.ys * g.zs;
    if (host_slots) {
        for (long long c = 0; c < ncell; c++)
            if (host_slots[c] > nmat) { err = "material slot above nmat"; return QMS_ERR_ARG; }
        CK(cudaMemcpyAsync(ids, host_slots, ncell, cudaMemcpyHostToDevice, st));
    }
    qms_fill_table(htab64, rows6, nmat);
    qms_fill_table(htab32, rows6, nmat);
    CK(cudaMemcpyAsync(dtab64, &htab64, sizeof(htab64), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dtab32, &htab32, sizeof(htab32), cudaMemcpyHostToDevice, st));
    // node coefficients, then the Jacobi diagonals (velocity does not enter the diagonal)
    qms_launch_node_coef<float>(g, coef32(), nc32, st);
    qms_launch_node_coef<double>(g, coef64(), nc64, st);
    if (nc16) qms_launch_coef_bf16(g, nc32, nc16, st);
    if (df_resid) qms_launch_split_flat(6 * qms_pl(g).comp, nc64, ncdf, st);
    if (rsg) qms_launch_rhs_coef(g, ids, dtab64, desc.dt, rsg, rsdt, st);
    if (dinvdf) qms_launch_dinv_df(g, coef64(), qms_step_par<double>(g, 0, 0, 0, desc.dt, true), dinvdf, st);
    rfin_ok = false;
    hist_len = 0;
    w_len = 0;
    last_chained = false;
    QCoef<float> c32 = coef32();
    qms_launch_diag_pl(g, c32, qms_step_par<float>(g, 0, 0, 0, desc.dt, false), dg_steady, st);
    qms_launch_diag_pl(g, c32, qms_step_par<float>(g, 0, 0, 0, desc.dt, true), dg_tr, st);
    CK(cudaGetLastError());
    if (use_mg) {
        const double vshift = desc.mg_vshift;
        for (int tr = 0; tr < 2; tr++) {
            int rc;
            if (fp64_inner) {
                QmsMG<double>& M = mgd[tr];
                M.nu1 = M.nu2 = desc.mg_sweeps; M.omega = desc.mg_omega; M.alpha = desc.mg_alpha;
                M.nu_coarse = desc.mg_coarse_sweeps;
                M.nu_v = desc.mg_v_sweeps;
                M.tail_points = desc.mg_tail_points;
                M.vcut = desc.mg_v_coarse_cut;
                rc = M.build(g, coef64(), qms_step_par<double>(g, 0, 0, 0, desc.dt, tr == 1), vshift, st);
                if (rc) { err = M.err; return QMS_ERR_CUDA; }
            } else {
                QmsMG<float>& M = mgf[tr];
                M.nu1 = M.nu2 = desc.mg_sweeps; M.omega = (float)desc.mg_omega; M.alpha = (float)desc.mg_alpha;
                M.nu_coarse = desc.mg_coarse_sweeps;
                M.nu_v = desc.mg_v_sweeps;
                M.tail_points = desc.mg_tail_points;
                M.vcut = desc.mg_v_coarse_cut;
                rc = M.build(g, coef32(), qms_step_par<float>(g, 0, 0, 0, desc.dt, tr == 1), (float)vshift, st);
                if (rc) { err = M.err; return QMS_ERR_CUDA; }
            }
        }
    }
    regions.release();
    if (use_mg) {
        // the region space needs the slots on the host
        std::vector<uint8_t> hslots;
        const uint8_t* sl = host_slots;
        if (!sl) {
            hslots.resize(ncell);
            CK(cudaMemcpyAsync(hslots.data(), ids, ncell, cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            sl = hslots.data();
        }
        const double cut = desc.mg_region_cut != 0.0 ? desc.mg_region_cut : (fp64_inner ? 1e-9 : 1e-6);
        if (cut > 0.0 && regions.build(g, sl, rows6, nmat, desc.mg_vshift, cut, st)) {
            err = regions.err;
            return QMS_ERR_CUDA;
        }
    }
    CK(cudaStreamSynchronize(st));
    return 0;
}

QCoef<float> QmsSolver::coef32() const { return QCoef<float>{g, ids, dtab32, (float)(1.0 / QMS_MU0), nc32}; }
QCoef<double> QmsSolver::coef64() const { return QCoef<double>{g, ids, dtab64, 1.0 / QMS_MU0, nc64}; }

int QmsSolver::finalize(int fop, int nsum, long long nb) {
    pdl_launch(qk_finalize, dim3(1), dim3(512), 0, st, 0, part, nb, nsum, S, fop, status);
    nlaunch++;
    return 0;
}

template <typename T>
void QmsSolver::op(bool adv, int mode, const QStepPar<T>& P, const T* xin, const T* bin, T* y, const T* w,
                   double* partials) {
    const double ncell = (double)g.xs * g.ys * g.zs;
    // the reference-layout operator serves the FP64 refinement residual (profile kind 3)
    OpEv* ev = prof_begin(mode == QOPH_RESID ? 3 : (sizeof(T) == 8 ? 1 : 0),
                          (double)g.n * sizeof(T) * (2 + (w && w != xin ? 1 : 0) + (bin ? 1 : 0)) + ncell);
    qms_launch_operator<T>(g, coef<T>(), P, adv, mode, xin, bin, y, w, partials, st);
    nlaunch++;
    prof_end(ev);
}
template void QmsSolver::op<float>(bool, int, const QStepPar<float>&, const float*, const float*, float*,
                                   const float*, double*);

const CUtensorMap& QmsSolver::tmap(const void* p) const { return tmaps.at(p); }
const CUtensorMap& QmsSolver::tmapq(const void* p, int qs) const {
    return qs == 1 ? tmapsA.at(p) : (qs == 2 ? tmapsV.at(p) : tmaps.at(p));
}

template <typename T>
void QmsSolver::op_pl(bool adv, QPlMode mode, const QStepPar<T>& P, const T* xin, T* y, const T* w, double* partials) {
    const double ncell = (double)g.xs * g.ys * g.zs;
    OpEv* ev = prof_begin(sizeof(T) == 8 ? 1 : 0, (double)g.n * sizeof(T) * (2 + (w && w != xin ? 1 : 0)) + ncell);
    qms_launch_op_pl<T>(g, P, mode == QPL_APPLY_A ? tmapq(xin, 1) : tmap(xin), sizeof(T) == 8 ? cmap64 : cmap32, adv, mode,
                        y, w, partials, status, st);
    nlaunch++;
    prof_end(ev);
}
template void QmsSolver::op_pl<float>(bool, QPlMode, const QStepPar<float>&, const float*, float*, const float*, double*);
template void QmsSolver::op_pl<double>(bool, QPlMode, const QStepPar<double>&, const double*, double*, const double*,
                                       double*);
template void QmsSolver::op<double>(bool, int, const QStepPar<double>&, const double*, const double*, double*,
                                    const double*, double*);

QmsSolver::OpEv* QmsSolver::prof_begin(int kind, double bytes) {
    if (!prof) return nullptr;
    if (evused == evpool.size()) {
        OpEv e{};
        cudaEventCreate(&e.a);
        cudaEventCreate(&e.b);
        evpool.push_back(e);
    }
    OpEv* ev = &evpool[evused++];
    ev->kind = kind;
    ev->bytes = bytes;
    cudaEventRecord(ev->a, st);                 // (a profiled solve captures nothing)
    return ev;
}

void QmsSolver::prof_end(OpEv* ev) {
    if (ev) cudaEventRecord(ev->b, st);
}

bool QmsSolver::prof_accum(const OpEv& e) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, e.a, e.b) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (e.kind == 1) { profacc.op64_launches++; profacc.op64_ms += ms; profacc.op64_bytes += e.bytes; }
    else if (e.kind == 0) { profacc.op32_launches++; profacc.op32_ms += ms; profacc.op32_bytes += e.bytes; }
    else if (e.kind == 3) { profacc.resid_launches++; profacc.resid_ms += ms; profacc.resid_bytes += e.bytes; }
    else if (e.kind == MGPROF_A_SWEEP) { profacc.mg0a_launches++; profacc.mg0a_ms += ms; profacc.mg0a_bytes += e.bytes; }
    else { profacc.mg_cycles++; profacc.mg_ms += ms; }
    return true;
}

int QmsSolver::profile_enable(bool on) {
    if (prof || on) {
        cudaStreamSynchronize(st);
    }
    prof = on;
    nlaunch = 0;
    evused = 0;
    profacc = qms_profile{};
    return 0;
}

int QmsSolver::profile_collect(qms_profile* out) {
    CK(cudaStreamSynchronize(st));
    for (size_t q = 0; q < evused; q++)
        if (!prof_accum(evpool[q])) { err = "profile events could not be timed"; return QMS_ERR_CUDA; }
    evused = 0;
    profacc.launches = nlaunch;
    *out = profacc;
    return 0;
}

int QmsSolver::read_scalars() {
    CK(cudaMemcpyAsync(hS, S, S_COUNT * 8, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return 0;
}

template <typename T>
void QmsSolver::precond(const T* r, const float* bscale, T* z, bool mask_v, bool transient, bool jacobi_pcg,
                        const QStepPar<T>* P, bool adv) {
    if (use_mg) {
        OpEv* ev = prof_begin(2, 0.0);
        const bool f32 = sizeof(T) == 4;
        // the cycles' level-0 tiles read the bf16 coefficients in an FP32 hierarchy
        const CUtensorMap& cm = f32 ? cmap16 : cmap64;
        auto cycle = [&](const T* b, int qs, const CUtensorMap& cmq) {
            // b's own tile map for the fused first sweeps of the subset cycles (a mapped vector)
            const CUtensorMap* bm = nullptr;
            if (qs != 0) {
                auto& tm = qs == 1 ? tmapsA : tmapsV;
                auto it = tm.find((const void*)b);
                if (it != tm.end()) bm = &it->second;
            }
            if (f32)
                nlaunch += mgf[transient ? 1 : 0].vcycle((const float*)b, bscale != nullptr, (float*)z, tmapq(z, qs),
                                                         mgtmp, tmapq(mgtmp, qs), cmq, status, st, qs, bm);
            else
                nlaunch += mgd[transient ? 1 : 0].vcycle((const double*)b, bscale != nullptr, (double*)z,
                                                         tmapq(z, qs), (double*)mgtmp, tmapq(mgtmp, qs), cmq, status,
                                                         st, qs);
        };
        if (P && !mask_v && bscale && desc.mg_coupling == 1) {
            // lower block-triangular: the A blocks first, then the V block on the residual that
            // the A correction leaves in the V rows (row-scaled like r)
            T* tv = (T*)mgtmp2;
            cycle(r, 1, cm);
            qms_launch_op_pl<T>(g, *P, tmapq(z, 1), f32 ? cmapV32 : cmapV64, adv, QPL_VCOUPLE, tv, r, nullptr,
                                status, st);
            cycle(tv, 2, f32 ? cmapV16 : cmapV64);
            nlaunch++;
            regions.apply<T>(tv, bscale, z, st, nlaunch);
        } else if (mask_v) {
            cycle(r, 1, cm);                     // z's V block stays as it is (zero)
        } else {
            cycle(r, 0, cm);
            regions.apply<T>(r, bscale, z, st, nlaunch);
        }
        prof_end(ev);
    } else if (jacobi_pcg) {
        qk_jacobi<T><<<(int)vec_blocks, 256, 0, st>>>(npl, mask_v ? 3 * qms_pl(g).comp : npl, r,
                                                        transient ? dg_tr : dg_steady, z);
        nlaunch++;
    }
}

template <typename T>
int QmsSolver::inner_bicgstab(bool adv, bool transient, const double v[3], int& iters) {
    const long long n = npl;
    T* r = (T*)vec[0]; T* rh = (T*)vec[1]; T* p = (T*)vec[2]; T* vv = (T*)vec[3];
    T* s = (T*)vec[4]; T* t = (T*)vec[5]; T* e = (T*)vec[6];
    // right preconditioner of the row-scaled operator D^-1 M: y = MG(D p); identity without MG
    T* y = use_mg ? (T*)vec[7] : p;
    T* z = use_mg ? (T*)vec[8] : s;
    const float* dg = transient ? dg_tr : dg_steady;
    QStepPar<T> P = qms_step_par<T>(g, v[0], v[1], v[2], desc.dt, transient);
    const int vb = (int)vec_blocks;
    resid_to_inner<T>(r);
    qk_bicg_init<T><<<vb, 256, 0, st>>>(n, r, rh, p, vv, e, part);
    nlaunch++;
    finalize(FIN_BICG_INIT, 1, vec_blocks);
    const double tol2 = desc.inner_rtol * desc.inner_rtol;
    iters = 0;
    for (int it = 0; it < desc.max_inner; it++) {
        qk_bicg_p<T><<<vb, 256, 0, st>>>(n, r, p, vv, S);
        nlaunch++;
        if (use_mg) precond<T>(p, dg, y, false, transient, false, &P, adv);
        op_pl<T>(adv, QPL_SCALED, P, y, vv, rh, part);
        finalize(FIN_BICG_ALPHA, 1, nbpl);
        qk_bicg_s<T><<<vb, 256, 0, st>>>(n, r, vv, s, S);
        nlaunch++;
        if (use_mg) precond<T>(s, dg, z, false, transient, false, &P, adv);
        op_pl<T>(adv, QPL_SCALED, P, z, t, s, part);
        finalize(FIN_BICG_OMEGA, 2, nbpl);
        qk_bicg_xr<T><<<vb, 256, 0, st>>>(n, y, z, s, t, rh, e, r, S, part);
        nlaunch++;
        finalize(FIN_BICG_RHO, 2, vec_blocks);
        iters = it + 1;
        if ((it + 1) % desc.check_every == 0 || it + 1 == desc.max_inner) {
            int rc = read_scalars();
            if (rc) return rc;
            if (!(hS[S_RR] <= tol2 * hS[S_RR0])) {
                unsigned stt = 0;
                CK(cudaMemcpyAsync(&stt, status, 4, cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                if (stt & QMS_ST_BREAKDOWN) break;
                continue;
            }
            break;
        }
    }
    qms_launch_ref_add_pl<T>(g, e, S + S_NRM, x, st);
    nlaunch++;
    CK(cudaGetLastError());
    return 0;
}


// FGMRES in three parts: the start of a cycle, its steps j0 <= j < j1, and its end after k steps
// (the small solve and the FP64 update of x)
template <typename T>
void QmsSolver::gmres_begin() {
    qk_gm_reset<<<1, 128, 0, st>>>(std::min(desc.gmres_m, GM_MAXM), gm_scal);
    resid_to_inner<T>((T*)gmV[0]);
    nlaunch++;
}

template <typename T>
void QmsSolver::gmres_steps(bool adv, bool transient, const double v[3], int j0, int j1) {
    const long long n = npl;
    const int m = std::min(desc.gmres_m, GM_MAXM);
    const float* dg = transient ? dg_tr : dg_steady;
    QStepPar<T> P = qms_step_par<T>(g, v[0], v[1], v[2], desc.dt, transient);
    // two packets per thread at least: fewer partial sums to add up on small grids
    const int vb = (int)std::max(1LL, std::min(vec_blocks, (n * (long long)sizeof(T) / 16 + 511) / 512));
    GmPtrs Vp{};
    for (int i = 0; i <= m; i++) Vp.p[i] = gmV[i];
    T* w = (T*)vec[0];
    for (int j = j0; j < j1; j++) {
        T* vj = (T*)gmV[j];
        T* zj = use_mg ? (T*)gmZ[j] : vj;
        if (use_mg) precond<T>(vj, dg, zj, false, transient, false, &P, adv);
        op_pl<T>(adv, QPL_SCALED, P, zj, w, nullptr, nullptr);
        nlaunch += gm_dots<T>(j + 1, vb, st, n, Vp, w, part, 0, j, m, gm_H, gm_scal, gm_count, nsm);
        nlaunch += gm_orth<T>(j + 1, vb, st, n, j, m, Vp, gm_H, 0, w, part, gm_scal, (T*)gmV[j + 1], gm_count, status, nsm);
        pdl_launch(qk_gm_scale<T>, dim3(std::min(vb, nsm)), dim3(256), 0, st, 0, n, w, (T*)gmV[j + 1], gm_scal);
        nlaunch++;
    }
}

template <typename T>
void QmsSolver::gmres_end(int k) {
    const int m = std::min(desc.gmres_m, GM_MAXM);
    GmPtrs Zp{};
    for (int i = 0; i < m; i++) Zp.p[i] = use_mg ? gmZ[i] : gmV[i];
    qk_gm_solve<<<1, 256, 0, st>>>(k, m, gm_H, gm_scal);
    nlaunch += 1 + gm_update<T>(k, st, g, m, Zp, gm_scal, S, x);
    last_gm_k = k;
}

int QmsSolver::gmres_estimate(double& est) {
    CK(cudaMemcpyAsync(hS, gm_scal, 8 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    est = hS[1] / hS[0];
    return 0;
}

// a cycle of fixed_k steps, or (fixed_k = 0) with a look at the estimate every check_every steps
template <typename T>
int QmsSolver::inner_gmres(bool adv, bool transient, const double v[3], int& iters, int fixed_k) {
    const int m = std::min(desc.gmres_m, GM_MAXM);
    const int kmax = fixed_k > 0 ? std::min(fixed_k, m) : m;
    gmres_begin<T>();
    int k = 0;
    while (k < kmax) {
        const int j1 = fixed_k > 0 ? kmax : std::min(kmax, k + desc.check_every);
        gmres_steps<T>(adv, transient, v, k, j1);
        k = j1;
        if (fixed_k <= 0) {
            double est;
            int rc = gmres_estimate(est);
            if (rc) return rc;
            if (!(est > desc.inner_rtol)) break;     // also stops on a non-finite estimate
        }
    }
    gmres_end<T>(k);
    iters = k;
    CK(cudaGetLastError());
    return 0;
}

static double wall_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// Steps j0 .. j0 + kSeg - 1 of a cycle as one CUDA graph, captured once per j0 for the operator of
// this solve and replayed; the operator of another velocity starts over.  Until then the steps are
// launched directly: kSegDirect times (a replay saves some 10 us over direct launches, a capture alone
// takes 0.2 to 0.7 ms), and for as long as captures would take more than an eighth of the time that the
// handle has spent in cycles.  Among 16 solves that share the driver's locks a capture takes 50 to 100 ms,
// up to 0.7 s while requests are being set up: first steps that captured all of their segments took up
// to 1.8 s.  24 requests at 50 ms, 99th percentile of a step with 10 (50) steps each: 1.1-1.8 s
// (0.38-0.46) with captures at once, 0.51-0.77 (0.43-0.62) so, 0.49-0.90 by the eighth alone, 0.51-0.64
// and 0.34-0.41 from 32 and 48 direct launches on.  Repeated runs of 48^3 take 2 and 5 % longer with
// the latter two; first runs on 16x14x12 and 32^3 take 3.5 and 2 % longer so than with captures at once.
int QmsSolver::gmres_segment(bool adv, bool transient, const double v[3], int j0, int j1, bool graph) {
    auto steps = [&] {
        if (fp64_inner) gmres_steps<double>(adv, transient, v, j0, j1);
        else gmres_steps<float>(adv, transient, v, j0, j1);
    };
    if (!graph) {
        steps();
        CK(cudaGetLastError());
        return 0;
    }
    if (!seg_valid || seg_tr != transient || seg_v[0] != v[0] || seg_v[1] != v[1] || seg_v[2] != v[2]) {
        drop_segments();
        seg_valid = true;
        seg_tr = transient;
        for (int q = 0; q < 3; q++) seg_v[q] = v[q];
    }
    const size_t at = (size_t)(j0 / kSeg);
    if (segs.size() <= at) segs.resize(at + 1);
    SegGraph& G = segs[at];
    if (!G.exec && (G.direct < kSegDirect || capture_s + capture_last_s > cycles_s / 8)) {
        G.direct = std::min(G.direct + 1, kSegDirect);
        steps();
        CK(cudaGetLastError());
        return 0;
    }
    if (!G.exec) {
        const double t0 = wall_s();
        const long long n0 = nlaunch;
        CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        steps();
        cudaGraph_t graph_ = nullptr;
        cudaError_t e = cudaStreamEndCapture(st, &graph_);
        if (e == cudaSuccess) e = cudaGraphInstantiate(&G.exec, graph_, 0);
        if (graph_) cudaGraphDestroy(graph_);
        G.launches = nlaunch - n0;
        nlaunch = n0;
        capture_last_s = wall_s() - t0;
        capture_s += capture_last_s;
        if (e != cudaSuccess) {
            cudaGetLastError();
            G.exec = nullptr;
            err = std::string("graph capture: ") + cudaGetErrorString(e);
            return QMS_ERR_CUDA;
        }
    }
    CK(cudaGraphLaunch(G.exec, st));
    nlaunch += G.launches;
    return 0;
}

// One cycle that ends when its residual estimate reaches `stop` (or the basis is full).  The first
// look at the estimate comes at 0.6 of the count that the last cycles' rate predicts (a look costs a
// host wait of some 15 us, a step too many 0.2 to 5 ms).  A cycle that ran on past the FP32 floor cost most: the counts
// that were learned across solves before grew to 32 steps where 8 reach it (a plate in harmonic
// motion: 84 steps per time step instead of 28).
int QmsSolver::gmres_cycle(bool adv, bool transient, const double v[3], double stop, bool graph, int& iters) {
    const int m = std::min(desc.gmres_m, GM_MAXM);
    const double t0 = wall_s();
    if (fp64_inner) gmres_begin<double>();
    else gmres_begin<float>();
    int k = 0, upto = kSeg;
    if (gm_rate < 0.0) upto = (int)std::min((double)m, 0.6 * std::log(stop) / gm_rate);
    upto = std::min(m, std::max(kSeg, upto));
    double est = 1.0;
    for (;;) {
        while (k < upto) {
            const int j1 = std::min(m, k + kSeg);
            int rc = gmres_segment(adv, transient, v, k, j1, graph);
            if (rc) return rc;
            k = j1;
        }
        int rc = gmres_estimate(est);
        if (rc) return rc;
        if (!(est > stop) || k >= m) break;          // also stops on a non-finite estimate
        upto = std::min(m, k + kSeg);
    }
    if (est > 0.0 && est < 1.0) {
        const double lr = std::log(est) / k;
        gm_rate = gm_rate < 0.0 ? 0.5 * (gm_rate + lr) : lr;
    }
    if (fp64_inner) gmres_end<double>(k);
    else gmres_end<float>(k);
    cycles_s += wall_s() - t0;
    iters = k;
    CK(cudaGetLastError());
    return 0;
}


template <typename T>
int QmsSolver::inner_pcg(bool transient, int& iters) {
    const long long n = npl;
    T* r = (T*)vec[0]; T* z = (T*)vec[1]; T* p = (T*)vec[2]; T* q = (T*)vec[3]; T* e = (T*)vec[6];
    const float* dg = transient ? dg_tr : dg_steady;
    QStepPar<T> P = qms_step_par<T>(g, 0, 0, 0, desc.dt, transient);
    const int vb = (int)vec_blocks;
    // V block frozen at zero: the steady magnetostatic system with v = 0 has V = 0.  The vectors' V parts
    // are left alone (z's and the correction e's are zero), and the cycles work on the A blocks.
    const long long nA = 3 * qms_pl(g).comp;
    resid_to_inner<T>(r);
    qk_cg_init<T><<<vb, 256, 0, st>>>(n, dg, r, e);
    nlaunch++;
    CK(cudaMemsetAsync(z + nA, 0, (n - nA) * sizeof(T), st));
    precond<T>(r, nullptr, z, true, transient, true);
    pdl_launch(qk_cg_dot<T>, dim3(vb), dim3(256), 0, st, 0, nA, r, z, p, part);
    nlaunch++;
    finalize(FIN_CG_INIT, 2, vec_blocks);
    const double tol2 = desc.inner_rtol * desc.inner_rtol;
    iters = 0;
    for (int it = 0; it < desc.max_inner; it++) {
        op_pl<T>(false, QPL_APPLY_A, P, p, q, p, part);
        finalize(FIN_CG_ALPHA, 1, nbpl);
        pdl_launch(qk_cg_axpy<T>, dim3(vb), dim3(256), 0, st, 0, nA, q, S, T(-1), r);
        nlaunch++;
        precond<T>(r, nullptr, z, true, transient, true);
        pdl_launch(qk_cg_dot<T>, dim3(vb), dim3(256), 0, st, 0, nA, r, z, nullptr, part);
        nlaunch++;
        finalize(FIN_CG_BETA, 2, vec_blocks);
        iters = it + 1;
        bool done = it + 1 == desc.max_inner;
        if ((it + 1) % desc.check_every == 0 || done) {
            int rc = read_scalars();
            if (rc) return rc;
            done = done || hS[S_RZ] <= tol2 * hS[S_RZ0];
        }
        if (done) pdl_launch(qk_cg_axpy<T>, dim3(vb), dim3(256), 0, st, 0, nA, p, S, T(1), e);
        else pdl_launch(qk_cg_ep<T>, dim3(vb), dim3(256), 0, st, 0, nA, z, p, e, S);
        nlaunch++;
        if (done) break;
    }
    qms_launch_ref_add_pl<T>(g, e, S + S_NRM, x, st);
    nlaunch++;
    CK(cudaGetLastError());
    return 0;
}

int QmsSolver::residual_launch(bool adv, bool transient, const double v[3], bool exact) {
    if (start_resid_ready && !exact) {
        // the step start (qk_step_start) formed this residual and its partials
        start_resid_ready = false;
        last_resid_df = true;
        finalize(FIN_RESID, 4, nbpl);
        return 0;
    } else if (df_resid && anchor_ready && anchor_is_residual && !exact) {
        // x is the anchor state: the residual is the anchor's
        OpEv* ev = prof_begin(3, (double)g.n * 8 * 3);
        qms_launch_anchor_resid(g, r0df, x, rpl, rfin, part, nbpl, st);
        nlaunch++;
        prof_end(ev);
        anchor_is_residual = false;
        last_resid_df = true;
    } else if (df_resid && anchor_ready && !exact) {
        // double-float from the anchor: dx = x - x0 split into the padded layout (with the |x|^2
        // partials), then the TMA-staged stencil on the FP32 pipe
        OpEv* ev = prof_begin(3, (double)g.n * 8 * 4 + (double)g.xs * g.ys * g.zs);
        qms_launch_delta_split(g, x, x0, xdf, part, nbpl, st);
        qms_launch_resid_df(g, qms_step_par<qdf>(g, v[0], v[1], v[2], desc.dt, transient), xdfmap, cdfmap, adv, rpl,
                            r0df, part, status, st, rfin);
        nlaunch += 2;
        prof_end(ev);
        last_resid_df = true;
    } else {
        QStepPar<double> P = qms_step_par<double>(g, v[0], v[1], v[2], desc.dt, transient);
        op<double>(adv, QOPH_RESID, P, x, b, r64, nullptr, part);
        if (df_resid && !exact) {
            // the anchor of the double-float residuals that follow in this solve (an exact
            // residual asked for between solves leaves the anchor and its chain as they are)
            qms_launch_split_ref_pl(g, r64, r0df, rpl, st);
            CK(cudaMemcpyAsync(x0, x, g.n * 8, cudaMemcpyDeviceToDevice, st));
            nlaunch++;
            anchor_ready = true;
        }
        last_resid_df = false;
        finalize(FIN_RESID, 4, nbop);
        return 0;
    }
    finalize(FIN_RESID, 4, nbpl);
    return 0;
}

template <typename T>
void QmsSolver::resid_to_inner(T* out) {
    if constexpr (sizeof(T) == 4) {
        if (df_resid) {
            qms_launch_pl_scale(npl, rpl, S + S_INVNRM, out, st);
            nlaunch++;
            return;
        }
    }
    qms_launch_pl_from_ref<T>(g, r64, S + S_INVNRM, out, st);
    nlaunch++;
}

// b of the last solve, formed from its start state (x0) when that solve took b - b_prev from
// the state difference instead
void QmsSolver::ensure_b() {
    if (b_fresh) return;
    qms_launch_rhs(g, ids, dtab64, last_ex, desc.dt, last_tr ? 1 : 0, x0, b, nullptr, st, rsg, rsdt);
    nlaunch++;
    b_fresh = true;
}

int QmsSolver::residual(bool adv, bool transient, const double v[3], bool exact) {
    int rc = residual_launch(adv, transient, v, exact);
    if (rc) return rc;
    CK(cudaGetLastError());
    return read_scalars();
}

void QmsSolver::drop_segments() {
    for (SegGraph& G : segs)
        if (G.exec) cudaGraphExecDestroy(G.exec);
    segs.clear();
    seg_valid = false;
}

void QmsSolver::drop_graphs() {
    drop_segments();
    for (StepGraph& G : sgraphs)
        if (G.exec) cudaGraphExecDestroy(G.exec);
    sgraphs.clear();
}

// One whole chained step as a graph (captured once per k, start variant and velocity, then
// replayed): returns after the step with the residual sums in hS and the cycles it ran.
int QmsSolver::step_graph(bool adv, const double v[3], const QStepStart& hs, bool wcalc, int k, int& cycles) {
    const bool dbx = hs.hx != nullptr;
    StepGraph* G = nullptr;
    for (StepGraph& e : sgraphs)
        if (e.k == k && e.xo == hs.xo && e.ls == hs.ls && e.wcalc == wcalc && e.dbx == dbx && e.v[0] == v[0] && e.v[1] == v[1] &&
            e.v[2] == v[2]) { G = &e; break; }
    if (!G) {
        // a run's counts fall from 13 to 3 or so: a cache of fewer than a run's graphs instantiated and
        // destroyed them all again in the next one (a destruction now and then held a step up by 50 ms)
        constexpr size_t kMax = 16;
        if (sgraphs.size() >= kMax) {
            size_t lru = 0;
            for (size_t q = 1; q < sgraphs.size(); q++) if (sgraphs[q].used < sgraphs[lru].used) lru = q;
            if (sgraphs[lru].exec) cudaGraphExecDestroy(sgraphs[lru].exec);
            sgraphs.erase(sgraphs.begin() + (long)lru);
        }
        StepGraph ng;
        cudaGraph_t graph = nullptr;
        CK(cudaGraphCreate(&graph, 0));
        cudaGraphConditionalHandle hc;
        cudaError_t e = cudaGraphConditionalHandleCreate(&hc, graph, 0, cudaGraphCondAssignDefault);
        const long long n0 = nlaunch;
        int rc = 0;
        if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(st, graph, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            cudaMemsetAsync(status, 0, 4, st);
            cudaMemcpyAsync(dptrs, hptrs, sizeof(QStepPtrs), cudaMemcpyHostToDevice, st);
            qms_launch_step_start(g, rfin, b, bprev, dinvdf, r0df, hs, rpl, part, nbpl, st, dptrs);
            finalize(FIN_RESID, 4, nbpl);
            qk_cond_init<<<1, 32, 0, st>>>(S, desc.tol, hc);
            nlaunch += 2;
            ng.pro = nlaunch - n0;
            // the conditional node at the end of the prologue
            cudaStreamCaptureStatus cs;
            cudaGraph_t cg = nullptr;
            const cudaGraphNode_t* deps = nullptr;
            size_t nd = 0;
            e = cudaStreamGetCaptureInfo(st, &cs, nullptr, &cg, &deps, nullptr, &nd);
            cudaGraphNodeParams cp = {};
            cp.type = cudaGraphNodeTypeConditional;
            cp.conditional.handle = hc;
            cp.conditional.type = cudaGraphCondTypeWhile;
            cp.conditional.size = 1;
            cudaGraphNode_t cn = nullptr;
            if (e == cudaSuccess) e = cudaGraphAddNode(&cn, cg, deps, nullptr, nd, &cp);
            if (e == cudaSuccess) e = cudaStreamUpdateCaptureDependencies(st, &cn, nullptr, 1, cudaStreamSetCaptureDependencies);
            cudaGraph_t got = nullptr;
            cudaError_t e2 = cudaStreamEndCapture(st, &got);
            if (e == cudaSuccess) e = e2;
            // the body: one refinement cycle and the test that sets the condition
            if (e == cudaSuccess) {
                cudaGraph_t body = cp.conditional.phGraph_out[0];
                e = cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
                if (e == cudaSuccess) {
                    const long long n1 = nlaunch;
                    int it = 0;
                    start_resid_ready = false;          // the body's residual is the double-float one
                    rc = inner_gmres<float>(adv, true, v, it, k);
                    if (rc == 0) rc = residual_launch(adv, true, v);
                    qk_cond_next<<<1, 32, 0, st>>>(S, desc.tol, kStepGraphCycles, hc);
                    nlaunch++;
                    ng.body = nlaunch - n1;
                    cudaGraph_t bg = nullptr;
                    e2 = cudaStreamEndCapture(st, &bg);
                    if (e == cudaSuccess) e = e2;
                }
            }
        }
        nlaunch = n0;
        if (rc == 0 && e == cudaSuccess) e = cudaGraphInstantiate(&ng.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (rc || e != cudaSuccess) {
            cudaGetLastError();
            if (ng.exec) cudaGraphExecDestroy(ng.exec);
            if (rc) return rc;
            err = std::string("step graph: ") + cudaGetErrorString(e);
            return QMS_ERR_CUDA;
        }
        ng.k = k; ng.xo = hs.xo; ng.ls = hs.ls; ng.wcalc = wcalc; ng.dbx = dbx;
        ng.v[0] = v[0]; ng.v[1] = v[1]; ng.v[2] = v[2];
        sgraphs.push_back(ng);
        G = &sgraphs.back();
    }
    // the rotating pointers of this step, read by the graph's copy node at launch
    *hptrs = QStepPtrs{hs.xo1, hs.xo2, hs.xo3, hs.wnew, hs.w1, hs.w2, hs.hx, b, bprev, hs.xo4, hs.w3};
    G->used = ++graph_clock;
    CK(cudaGraphLaunch(G->exec, st));
    int rc = read_scalars();                    // synchronises the stream
    if (rc) return rc;
    cycles = (int)hS[S_CYC];
    nlaunch += G->pro + (long long)cycles * G->body;
    last_resid_df = true;
    start_resid_ready = false;
    return 0;
}

// The inner vectors' padding and the Dirichlet rows beyond the tiles are zero and read by the sums over
// whole vectors, and no kernel of a solve writes them but in such a sum's wake: a projection that is not
// finite puts NaN there, where 0 * NaN would end every later solve too.
int QmsSolver::clear_inner() {
    auto clear = [&](void* p, size_t es) { return p ? cudaMemsetAsync(p, 0, npl * es, st) : cudaSuccess; };
    for (void* p : vec) CK(clear(p, tsize));
    for (void* p : gmV) CK(clear(p, tsize));
    for (void* p : gmZ) CK(clear(p, tsize));
    CK(clear(mgtmp, tsize));
    CK(clear(mgtmp2, tsize));
    CK(clear(rpl, 4));
    for (qdf* p : {xdf, r0df, rfin, wh[0], wh[1], wh[2], wh[3]}) CK(clear(p, 8));
    return 0;
}

int QmsSolver::solve(bool transient, const double v[3], const double B[3], const double G[9]) {
    CK(cudaSetDevice(dev));
    QmsExcite ex;
    for (int q = 0; q < 3; q++) { ex.B[q] = B[q]; ex.v[q] = v[q]; }
    for (int q = 0; q < 9; q++) ex.G[q] = G[q];
    // the previous solve's final residual anchors this one when the operator is the same
    const bool chain = df_resid && transient && rfin_ok && chain_len < QMS_CHAIN_MAX && chain_v[0] == v[0] &&
                       chain_v[1] == v[1] && chain_v[2] == v[2];
    // the start of a transient solve that follows solves with the same operator: an extrapolation
    // of the last solutions (x = hist[0], the one before in hist[1], ...), independent of how the
    // residual is anchored
    const bool same_op = transient && chain_v[0] == v[0] && chain_v[1] == v[1] && chain_v[2] == v[2];
    if (!same_op) hist_len = 0;
    // order of the extrapolation: the known solutions (hist_len, x_n included) less one
    int xo = !same_op || !xold ? 0 : std::max(0, std::min(std::min(desc.extrapolate, 3), hist_len - 1));
    bool same_field = true;
    for (int q = 0; q < 3; q++) same_field = same_field && chain_B[q] == B[q];
    for (int q = 0; q < 9; q++) same_field = same_field && chain_G[q] == G[q];
    field_run = same_field ? field_run + 1 : 1;
    // w_n = D^-1 M (x_n - x_{n-1}) follows when this solve and the last one are chained; the
    // residual of the extrapolated start then follows from the w of the last xo steps when the
    // Dirichlet values did not change over them
    const bool wcalc = chain && last_chained && wh[0];
    // the least-squares start over ls of the last state differences: the known solutions less
    // one, the stored residual images of the differences before d_n plus the one formed now,
    // and the solves with the same Dirichlet values all bound it
    int ls = 0;
    if (wcalc && same_op && xold && desc.start_ls > 0)
        ls = std::max(0, std::min(std::min(desc.start_ls, hist_len - 1), std::min(w_len + 1, field_run - 2)));
    if (ls > 0) xo = ls;
    const bool start_fused = wcalc && xo > 0 && w_len >= xo - 1 && field_run >= xo + 2;
    // with the field unchanged and x_(n-1) known, the anchor takes b - b_prev from x_n - x_(n-1)
    // (the step start, in double-float) and this solve forms no FP64 right-hand side
    const bool db_from_x = chain && same_field && hist_len >= 2 && hist_x && xold && rsg;
    start_resid_ready = false;
    // the whole step as one graph: a chained step whose start also forms the first residual, with
    // replayed refinement cycles of a known count (no profile events inside: they cannot live in
    // a conditional body)
    const bool use_step_graph = desc.use_graphs && desc.krylov == QMS_KRYLOV_GMRES && start_fused && db_from_x &&
                                gm_k_est > 0 && !prof && !trace && hptrs && !(desc.tol_v > 0.0);
    QStepStart sg_hs{};
    bool sg_wcalc = false;
    if (chain && !db_from_x) {
        ensure_b();                // b_prev: the last solve's right-hand side
        // x0 is copied, not swapped: the captured refinement graphs hold its address
        CK(cudaMemcpyAsync(x0, x, g.n * 8, cudaMemcpyDeviceToDevice, st));   // the previous solution
        std::swap(b, bprev);
    }
    last_ex = ex;
    last_tr = transient;
    if (!db_from_x) {
        // b from the previous solution (x); Dirichlet values written into x (warm start keeps them exact)
        qms_launch_rhs(g, ids, dtab64, ex, desc.dt, transient ? 1 : 0, x, b, x, st, rsg, rsdt);
        nlaunch++;
        b_fresh = true;
    } else {
        b_fresh = false;           // formed from x0 when asked for (ensure_b)
    }
    anchor_ready = false;          // the first residual of this solve is the FP64 anchor ...
    anchor_is_residual = false;
    if (chain) {                   // ... unless it follows from the previous one
        // the anchor, w_n and the extrapolated start in one pass; the residual of that start too
        // when start_fused (otherwise the double-float residual from the anchor follows)
        const int nw = nwh;                                     // w buffers: w_(n-1), w_(n-2), ..., the new one
        QStepStart hs{x,    xold, xold2, xold3, xo, wcalc ? wh[nw - 1] : nullptr, wh[0], wh[1],
                      db_from_x ? hist_x : nullptr, rsg, rsdt, desc.dt, db_from_x ? x0 : nullptr,
                      xold4, wh[2], ls, lsp, lsg};
        if (use_step_graph) {
            sg_hs = hs;                  // launched inside the step's graph below
            sg_wcalc = wcalc;
        } else {
            OpEv* ev = start_fused ? prof_begin(3, (double)g.n * (ls > 0 ? 8 * 11 + 8 * (ls - 1) + 8 * (2 * ls + 5) + 4
                                                                         : 8 * 11 + 8 * 2 * xo + 4)) : nullptr;
            qms_launch_step_start(g, rfin, b, bprev, dinvdf, r0df, hs, start_fused ? rpl : nullptr, part, nbpl, st);
            nlaunch++;
            prof_end(ev);
        }
        if (wcalc) {               // wh[0]: w_n, wh[1]: w_(n-1), the oldest becomes the next one's buffer
            qdf* fresh = wh[nw - 1];
            for (int q = nw - 1; q > 0; q--) wh[q] = wh[q - 1];
            wh[0] = fresh;
        }
        w_len = wcalc ? std::min(w_len + 1, std::max(1, nw - 1)) : 0;
        anchor_ready = true;
        chain_len++;
        // same field and no extrapolation: the Dirichlet values did not move, x is the anchor state
        anchor_is_residual = same_field && xo == 0;
        start_resid_ready = start_fused;
    } else {
        chain_len = 0;
        w_len = 0;
        if (xo > 0) {
            // the extrapolated start (Dirichlet rows keep the values just written); its residual
            // is the FP64 anchor
            qms_launch_extrapolate(g, x, xold, xold2, xold3, xo, st);
            nlaunch++;
        }
    }
    last_chained = chain;
    rfin_ok = false;
    if (!use_step_graph) CK(cudaMemsetAsync(status, 0, 4, st));
    const bool adv = v[0] != 0.0 || v[1] != 0.0 || v[2] != 0.0;
    const bool use_cg = !transient && !adv;
    stats = qms_stats{};
    double rel = INFINITY, prev_rn = INFINITY, sref = 0.0;
    int outer = 0, stalled = 0;
    graph_resid_ready = false;
    const int gm_m = std::min(desc.gmres_m, GM_MAXM);
    int graph_k_used = 0;                 // k of the step graph's cycle that produced this residual (0: none)
    int gm_cycles = 0;                    // FGMRES cycles run in this solve
    int graph_cycles = 0;                 // ... of them in the step's graph
    double best_rn = INFINITY, best_rel = INFINITY;
    if (use_step_graph) {
        // the step (start and up to kStepGraphCycles cycles) in one graph; the loop below takes
        // over from the residual it leaves, as after a replayed cycle
        int cyc = 0;
        int rc = step_graph(adv, v, sg_hs, sg_wcalc, gm_k_est, cyc);
        if (rc) return rc;
        graph_resid_ready = true;
        stats.step_graph = 1;
        stats.initial_residual = hS[S_REL0];
        if (cyc > 0) {
            outer = cyc;
            sref = hS[S_SREF];
            prev_rn = hS[S_PRN_LAST];
            graph_k_used = gm_k_est;
            gm_cycles = graph_cycles = cyc;
            stats.inner_iterations = cyc * gm_k_est;
            last_inner = 2;
            last_gm_k = gm_k_est;
        }
    }
    for (;;) {
        int rc = 0;
        if (!graph_resid_ready) {
            rc = residual(adv, transient, v);
            if (rc) return rc;
        }
        graph_resid_ready = false;
        const double xn = std::sqrt(hS[S_XA] + hS[S_XV]);
        const double rn = std::sqrt(hS[S_RA] + hS[S_RV]);
        // The scale is fixed by the state at the start of the solve (the previous step, or the
        // Dirichlet values for the steady state): a correction that blew up x must not make
        // ||r|| / ||x|| look small.
        if (outer == 0) sref = xn > 0 ? xn : 1.0;
        const double scale = std::min(std::max(xn, sref), 100.0 * sref);
        rel = rn / scale;
        if (outer == 0) stats.initial_residual = rel;
        if (!std::isfinite(rel)) { stats.status |= QMS_ST_NAN; break; }
        // optionally the potential block on its own scale as well: where |x| is dominated by A
        // (slow fields, small potentials), rel alone does not bound V's relative error
        const bool v_ok = !(desc.tol_v > 0.0) || hS[S_XV] == 0.0 ||
                          std::sqrt(hS[S_RV]) <= desc.tol_v * std::sqrt(hS[S_XV]);
        if ((rel <= desc.tol && v_ok) || rn == 0.0) break;
        // a cycle of the step's graph that gained less than a tenth with a short basis is not a stall
        const bool k_limited = graph_k_used > 0 && graph_k_used < gm_m && rn < prev_rn && rn > 0.1 * prev_rn;
        graph_k_used = 0;
        // Stall: near the round-off floor (within 1e3 of the tolerance) two iterations without
        // halving the residual end the solve; elsewhere only three iterations that gain less
        // than 10 % do, so that slowly but steadily converging solves continue.
        const bool near_floor = rel <= 1e3 * desc.tol;
        const bool slow = near_floor ? rn > 0.5 * prev_rn : rn > 0.9 * prev_rn;
        stalled = slow && !k_limited ? stalled + 1 : 0;
        if (stalled >= (near_floor ? 2 : 3)) {
            if (rel > 1e3 * desc.tol) stats.status |= QMS_ST_NO_CONVERGENCE;
            break;
        }
        // best state so far: a hard solve may lose ground for an iteration or two before it
        // gains again; whatever ends the solve, it ends at the best iterate
        if (rn < best_rn) {
            best_rn = rn;
            best_rel = rel;
            CK(cudaMemcpyAsync(xbest, x, g.n * 8, cudaMemcpyDeviceToDevice, st));
        }
        if (trace) {
            double est = 0.0;
            if (outer > 0 && last_inner == 2) {
                CK(cudaMemcpyAsync(hS + S_COUNT - 2, gm_scal, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                est = hS[S_COUNT - 1] / hS[S_COUNT - 2];
            }
            std::fprintf(stderr, "qms: %s outer %d |r| %.3e rel %.3e |x| %.3e |rA| %.3e |rV| %.3e inner-est %.2e k %d\n",
                         transient ? "step" : "steady", outer, rn, rel, xn, std::sqrt(hS[S_RA]), std::sqrt(hS[S_RV]),
                         est, last_gm_k);
        }
        if (outer >= desc.max_outer) { stats.status |= QMS_ST_NO_CONVERGENCE; break; }
        prev_rn = rn;
        int it = 0;
        if (use_cg) {
            last_inner = 0;
            rc = fp64_inner ? inner_pcg<double>(transient, it) : inner_pcg<float>(transient, it);
        } else if (desc.krylov == QMS_KRYLOV_BICGSTAB) {
            last_inner = 1;
            rc = fp64_inner ? inner_bicgstab<double>(adv, transient, v, it)
                            : inner_bicgstab<float>(adv, transient, v, it);
        } else if (desc.use_graphs) {
            // The reduction still wanted (to a tenth of the tolerance), in as few equal cycles as
            // inner_rtol allows: the FP32 inner solve gains little past ~1e-3 per cycle (its own
            // rounding), so deeper cycles buy less than a restart from a fresh residual
            last_inner = 2;
            const double want = std::log(std::min(0.1, 0.1 * desc.tol / rel));
            const double most = std::log(std::min(0.5, std::max(desc.inner_rtol, 1e-12)));
            const double stop = std::exp(want / std::max(1.0, std::ceil(want / most)));
            // replayed from graphs once the operator is that of the solve before (a motion that
            // changes it every step would pay a capture per step)
            rc = gmres_cycle(adv, transient, v, stop, same_op && !prof, it);
            gm_cycles++;
        } else {
            last_inner = 2;
            rc = fp64_inner ? inner_gmres<double>(adv, transient, v, it, 0) : inner_gmres<float>(adv, transient, v, it, 0);
            gm_cycles++;
        }
        if (rc) return rc;
        stats.inner_iterations += it;
        outer++;
    }
    // the final residual (rfin) anchors the next transient solve when it belongs to the state
    // that this solve leaves in x
    rfin_ok = df_resid && transient && last_resid_df && rel <= desc.tol;
    // history of converged transient solutions for the extrapolated start (x itself is the newest;
    // xold and xold2 the two before, rotated by pointer: only the extrapolation reads them)
    if (transient && rel <= desc.tol && xold) {
        double* freed = xold4 ? xold4 : xold3 ? xold3 : xold2 ? xold2 : xold;
        if (xold4) xold4 = xold3;
        if (xold3) xold3 = xold2;
        if (xold2) xold2 = xold;
        xold = hist_x;
        hist_x = freed;
        CK(cudaMemcpyAsync(hist_x, x, g.n * 8, cudaMemcpyDeviceToDevice, st));
        hist_len = std::min(hist_len + 1, xold4 ? 5 : xold3 ? 4 : xold2 ? 3 : 2);
    } else {
        hist_len = 0;
        last_chained = false;
    }
    for (int q = 0; q < 3; q++) { chain_v[q] = v[q]; chain_B[q] = B[q]; }
    for (int q = 0; q < 9; q++) chain_G[q] = G[q];
    if (!(rel <= desc.tol) && best_rel < rel && std::isfinite(best_rel)) {
        rfin_ok = false;
        CK(cudaMemcpyAsync(x, xbest, g.n * 8, cudaMemcpyDeviceToDevice, st));
        rel = best_rel;
        if (rel <= desc.tol) stats.status &= ~(unsigned)QMS_ST_NO_CONVERGENCE;
    }
    // FGMRES steps per cycle of a step run as one graph (its count is fixed when it is captured).
    // Solves with host-checked cycles leave the count that their reduction per FGMRES step says
    // reaches tol / 4 from their start, at most 12.  In the graph the start residual is within a few times the tolerance
    // and falls from step to step, so the count follows the measured rate: a one-cycle solve that
    // ended below tol / 4 takes the count that this solve's reduction per FGMRES step says reaches
    // tol / 4 from its start (at least one less); a solve that needed a second cycle goes up by one
    // (two after a third), and when its start had every direction it holds there for 4 solves (the
    // first steps of a run know fewer directions and start worse: floors from them kept the count
    // high well after).
    // (On steps 6-25 of the moving plate at 256^3, targets of tol / 10, tol / 4 and tol / 2 ran
    // 26.80, 25.51 and 24.74 ms per step; tol / 2 left the field 1.05e-8 from the plain FP64
    // solve's at one step of 200, tol / 4 at most 9.8e-9.)
    auto count_for = [&](double steps) {
        const double r0 = stats.initial_residual, goal = desc.tol / 4.0;
        if (!(r0 > goal && rel > 0.0 && r0 > rel)) return 1;
        // (r0 may be an ulp above rel: no reduction to speak of)
        const double per = std::log(r0 / rel) / std::max(1.0, steps), all = std::log(r0 / goal);
        return per * GM_MAXM > all ? (int)std::ceil(all / per) : GM_MAXM;
    };
    if (graph_cycles > 0 && rel <= desc.tol) {
        if (gm_ls_floor > 0 && ++gm_ls_floor_age > 4) { gm_ls_floor = 0; gm_ls_floor_age = 0; }
        if (gm_cycles >= 2) {
            gm_k_est = std::min(gm_m, gm_k_est + (gm_cycles >= 3 ? 2 : 1));
            if (ls >= desc.start_ls) {
                gm_ls_floor = gm_k_est;
                gm_ls_floor_age = 0;
            }
        } else if (rel < desc.tol / 4.0) {
            gm_k_est = std::max(std::max(1, gm_ls_floor), std::min(gm_k_est - 1, count_for(gm_k_est)));
        }
    } else if (transient && gm_cycles > 0 && rel <= desc.tol) {
        gm_k_est = std::min(std::min(gm_m, 12), std::max(2, count_for(stats.inner_iterations)));
        gm_ls_floor = 0;
    }
    unsigned stt = 0;
    double lsv[8] = {};
    CK(cudaMemcpyAsync(&stt, status, 4, cudaMemcpyDeviceToHost, st));
    if (ls > 0) CK(cudaMemcpyAsync(lsv, lsg, sizeof(lsv), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (ls > 0) {
        stats.start_ls = ls;
        for (int q = 0; q < 4; q++) stats.start_coef[q] = lsv[q];
        stats.start_base = lsv[4];
        stats.start_pred = lsv[5];
    }
    stats.status |= stt & ~(unsigned)QMS_ST_BREAKDOWN;
    stats.outer_iterations = outer;
    stats.final_residual = rel;
    if (stats.status & QMS_ST_NAN) return clear_inner();
    return 0;
}

// the operator's rows on vectors in the reference's order, through work vectors (zero again afterwards)
template <typename T>
int QmsSolver::apply_inner(int rows, bool transient, const double v[3], const double* dx, const double* dw,
                           double* dy) {
    const bool adv = rows != QMS_ROWS_A && (v[0] != 0.0 || v[1] != 0.0 || v[2] != 0.0);
    const QStepPar<T> P = qms_step_par<T>(g, adv ? v[0] : 0.0, adv ? v[1] : 0.0, adv ? v[2] : 0.0, desc.dt, transient);
    T* xi = (T*)vec[1];
    T* wi = (T*)vec[2];
    T* yi = (T*)vec[3];
    CK(cudaMemsetAsync(yi, 0, npl * sizeof(T), st));
    qms_launch_pl_from_ref<T>(g, dx, nullptr, xi, st);
    if (rows == QMS_ROWS_COUPLE) {
        qms_launch_pl_from_ref<T>(g, dw, nullptr, wi, st);
        qms_launch_op_pl<T>(g, P, tmapq(xi, 1), sizeof(T) == 4 ? cmapV32 : cmapV64, adv, QPL_VCOUPLE, yi, wi, nullptr,
                            status, st);
    } else {
        op_pl<T>(adv, rows == QMS_ROWS_A ? QPL_APPLY_A : QPL_SCALED, P, xi, yi, nullptr, nullptr);
    }
    CK(cudaMemsetAsync(dy, 0, g.n * sizeof(double), st));
    qms_launch_ref_add_pl<T>(g, yi, nullptr, dy, st);
    for (void* p : {vec[1], vec[2], vec[3]}) CK(cudaMemsetAsync(p, 0, npl * sizeof(T), st));
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(st));
    return 0;
}
template int QmsSolver::apply_inner<float>(int, bool, const double*, const double*, const double*, double*);
template int QmsSolver::apply_inner<double>(int, bool, const double*, const double*, const double*, double*);

int QmsSolver::fields(int which, int axis, int index, double* host_out) {
    CK(cudaSetDevice(dev));
    const long long ncell = (long long)g.xs * g.ys * g.zs;
    if (which == QMS_FIELD_CUBES) {
        qms_launch_hfield(g, ids, dtab64, x, H, H + ncell, H + 2 * ncell, st);
        nlaunch++;
        CK(cudaMemcpyAsync(host_out, H, 3 * ncell * 8, cudaMemcpyDeviceToHost, st));
    } else {
        int lim = axis == 0 ? g.xs : axis == 1 ? g.ys : g.zs;
        if (axis < 0 || axis > 2 || index < 1 || index > lim) { err = "slice axis/index out of range"; return QMS_ERR_ARG; }
        // only the slice's cells (what the reference dumps every step)
        qms_launch_hslice(g, ids, dtab64, x, axis, index, slicebuf, st);
        nlaunch++;
        long long m = (long long)(axis == 0 ? g.ys : g.xs) * (axis == 2 ? g.ys : g.zs);
        CK(cudaMemcpyAsync(host_out, slicebuf, 3 * m * 8, cudaMemcpyDeviceToHost, st));
    }
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(st));
    return 0;
}

int QmsSolver::fields_async(int which, int axis, int index, double* host_out, int slot) {
    CK(cudaSetDevice(dev));
    if (slot < 0 || slot >= kFieldSlots) { err = "field slot out of range"; return QMS_ERR_ARG; }
    const long long ncell = (long long)g.xs * g.ys * g.zs;
    long long m = 3 * ncell;
    if (which == QMS_FIELD_SLICE) {
        int lim = axis == 0 ? g.xs : axis == 1 ? g.ys : g.zs;
        if (axis < 0 || axis > 2 || index < 1 || index > lim) { err = "slice axis/index out of range"; return QMS_ERR_ARG; }
        m = 3LL * (axis == 0 ? g.ys : g.xs) * (axis == 2 ? g.ys : g.zs);
    } else if (which != QMS_FIELD_CUBES) {
        err = "unknown field kind";
        return QMS_ERR_ARG;
    }
    if (!cst) CK(cudaStreamCreateWithFlags(&cst, cudaStreamNonBlocking));
    if (!fev_ready[slot]) {
        CK(cudaEventCreateWithFlags(&fev_ready[slot], cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&fev_done[slot], cudaEventDisableTiming));
    }
    // the slot's previous copy must be finished before its device buffer is reused
    CK(cudaEventSynchronize(fev_done[slot]));
    if (fbuf_n[slot] < (size_t)m) {
        if (fbuf[slot]) CK(cudaFree(fbuf[slot]));
        fbuf[slot] = nullptr;
        fbuf_n[slot] = 0;
        CK(cudaMalloc(&fbuf[slot], m * 8));
        fbuf_n[slot] = (size_t)m;
    }
    double* d = fbuf[slot];
    if (which == QMS_FIELD_CUBES)
        qms_launch_hfield(g, ids, dtab64, x, d, d + ncell, d + 2 * ncell, st);
    else
        qms_launch_hslice(g, ids, dtab64, x, axis, index, d, st);
    nlaunch++;
    CK(cudaGetLastError());
    CK(cudaEventRecord(fev_ready[slot], st));
    CK(cudaStreamWaitEvent(cst, fev_ready[slot], 0));
    CK(cudaMemcpyAsync(host_out, d, m * 8, cudaMemcpyDeviceToHost, cst));
    CK(cudaEventRecord(fev_done[slot], cst));
    return 0;
}

int QmsSolver::fields_sync(int slot) {
    if (slot < 0 || slot >= kFieldSlots) return QMS_ERR_ARG;
    if (!fev_done[slot]) return 0;
    cudaError_t e = cudaEventSynchronize(fev_done[slot]);
    return e == cudaSuccess ? 0 : QMS_ERR_CUDA;
}

template int QmsSolver::inner_bicgstab<float>(bool, bool, const double*, int&);
template int QmsSolver::inner_bicgstab<double>(bool, bool, const double*, int&);
template int QmsSolver::inner_pcg<float>(bool, int&);
template int QmsSolver::inner_pcg<double>(bool, int&);
template int QmsSolver::inner_gmres<float>(bool, bool, const double*, int&, int);
template int QmsSolver::inner_gmres<double>(bool, bool, const double*, int&, int);
template void QmsSolver::precond<float>(const float*, const float*, float*, bool, bool, bool,
                                        const QStepPar<float>*, bool);
template void QmsSolver::precond<double>(const double*, const float*, double*, bool, bool, bool,
                                         const QStepPar<double>*, bool);
