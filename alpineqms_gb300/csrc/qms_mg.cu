// qms_mg.cu -- block-diagonal multigrid preconditioner for the Yee A-V system.
//
// The preconditioner treats the four unknown blocks (Ax, Ay, Az on edges, V on
// nodes) as four scalar 7-point problems: for each A component the
// same-direction couplings of its own row (curl-curl + gauge penalty
// coefficients 1/(mu h^2), F:476-525, F:682-731, F:888-937) plus the sigma/dt
// edge mass (F:1500-1504); for V the sigma-weighted Laplacian (F:1236-1285)
// with its diagonal shifted by a relative 1e-5: an isolated conductor's
// potential is fixed only through the 1e-12 S/m floor, a mode ~19 decades
// below the conductor scale that an exact inverse would amplify without bound.  Cross-component, advective and A-V
// coupling terms are left to the outer Krylov method.  For constant
// coefficients the A-block symbol |xi|^2 I - xi xi^T + diag(xi^2) lies
// between 1/3 and 2 times the vector Laplacian's, so the block-diagonal
// Laplacian preconditioner is spectrally equivalent.
//
// Hierarchy: unsmoothed 2x2x2 aggregation on each block's structured grid
// (general sizes; the two-layer Dirichlet shell leaves 253/254-point
// interiors that are not powers of two).  With piecewise-constant
// prolongation the Galerkin coarse operator of a 7-point operator is again
// 7-point: a coarse link is the sum of the fine links crossing between the two
// aggregates and a coarse diagonal is the sum of the fine diagonals minus
// twice the internal links.  All four blocks of a level are stored back to
// back and processed by one launch through a packed block-descriptor table.
// Smoother: weighted Jacobi.  Coarsest level: dense FP64 inverse per block.
#include "qms_mg.h"
#include "qms_pdl.cuh"
#include "qms_pl.h"
#include "qms_tile.cuh"

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <type_traits>
#include <vector>

namespace cg = cooperative_groups;

namespace {

// (i, j, k) of offset q in a block of n1 x n2 x n3 points, in 32-bit arithmetic (a block of a
// level holds far fewer than 2^32 points)
__device__ __forceinline__ void mg_ijk(long long q, int n1, int n2, int& i, int& j, int& k) {
    const unsigned u = (unsigned)q, a = u / (unsigned)n1, c = a / (unsigned)n2;
    i = (int)(u - a * (unsigned)n1);
    j = (int)(a - c * (unsigned)n2);
    k = (int)c;
}

template <typename T>
__device__ __forceinline__ int find_block(const MGLevelDev<T>& L, long long t) {
    int b = 0;
#pragma unroll
    for (int q = 1; q < MG_MAX_BLOCKS; q++)
        if (q < L.nb && t >= L.blk[q].off) b = q;
    return b;
}

// ---------------------------------------------------------------- fine level
// links (+1 neighbour along each axis), diagonal and activity of fine point
// (i, j, k) (1-based) of block b
template <typename T>
__device__ __forceinline__ bool mg_fine_point(const QGrid& g, const QCoef<T>& c, const QStepPar<T>& P, T vshift,
                                              int b, int i, int j, int k, T& w1, T& w2, T& w3, T& d) {
    bool active;
    w1 = w2 = w3 = T(0);
    d = T(1);
    if (b == 0) {            // Ax
        active = !qFixX(g, i, j, k);
        w1 = i < g.xs ? c.imux(i, j, k) * P.idx2 : T(0);
        w2 = j < g.Ny ? c.imuz(i, j, k) * P.idy2 : T(0);
        w3 = k < g.Nz ? c.imuy(i, j, k) * P.idz2 : T(0);
        if (active)
            d = (c.imuz(i, j, k) + c.imuz(i, j - 1, k)) * P.idy2 + (c.imuy(i, j, k) + c.imuy(i, j, k - 1)) * P.idz2 +
                (c.imux(i, j, k) + c.imux(i - 1, j, k)) * P.idx2 + c.sgx(i, j, k) * P.idt;
    } else if (b == 1) {     // Ay
        active = !qFixY(g, i, j, k);
        w1 = i < g.Nx ? c.imuz(i, j, k) * P.idx2 : T(0);
        w2 = j < g.ys ? c.imuy(i, j, k) * P.idy2 : T(0);
        w3 = k < g.Nz ? c.imux(i, j, k) * P.idz2 : T(0);
        if (active)
            d = (c.imuz(i, j, k) + c.imuz(i - 1, j, k)) * P.idx2 + (c.imux(i, j, k) + c.imux(i, j, k - 1)) * P.idz2 +
                (c.imuy(i, j, k) + c.imuy(i, j - 1, k)) * P.idy2 + c.sgy(i, j, k) * P.idt;
    } else if (b == 2) {     // Az
        active = !qFixZ(g, i, j, k);
        w1 = i < g.Nx ? c.imuy(i, j, k) * P.idx2 : T(0);
        w2 = j < g.Ny ? c.imux(i, j, k) * P.idy2 : T(0);
        w3 = k < g.zs ? c.imuz(i, j, k) * P.idz2 : T(0);
        if (active)
            d = (c.imuy(i, j, k) + c.imuy(i - 1, j, k)) * P.idx2 + (c.imux(i, j, k) + c.imux(i, j - 1, k)) * P.idy2 +
                (c.imuz(i, j, k) + c.imuz(i, j, k - 1)) * P.idz2 + c.sgz(i, j, k) * P.idt;
    } else {                 // V: the operator's own floor, diagonal shifted by (1 + vshift)
        const T fl = P.sigfloor;
        active = !qFixV(g, i, j, k);
        w1 = i < g.Nx ? fmax(c.sgx(i, j, k), fl) * P.idx2 : T(0);
        w2 = j < g.Ny ? fmax(c.sgy(i, j, k), fl) * P.idy2 : T(0);
        w3 = k < g.Nz ? fmax(c.sgz(i, j, k), fl) * P.idz2 : T(0);
        if (active)
            d = ((fmax(c.sgx(i, j, k), fl) + fmax(c.sgx(i - 1, j, k), fl)) * P.idx2 +
                 (fmax(c.sgy(i, j, k), fl) + fmax(c.sgy(i, j - 1, k), fl)) * P.idy2 +
                 (fmax(c.sgz(i, j, k), fl) + fmax(c.sgz(i, j, k - 1), fl)) * P.idz2) * (T(1) + vshift);
    }
    return active;
}

__device__ __forceinline__ bool mg_fine_active(const QGrid& g, int b, int i, int j, int k) {
    return b == 0 ? !qFixX(g, i, j, k) : b == 1 ? !qFixY(g, i, j, k) : b == 2 ? !qFixZ(g, i, j, k) : !qFixV(g, i, j, k);
}

// -------------------------------------------------------------- coarsening
// coarse point (I,J,K) aggregates fine points (2I..2I+1, 2J..2J+1, 2K..2K+1) (0-based):
// a coarse link is the sum of the fine links crossing between two aggregates, a
// coarse diagonal the sum of the fine diagonals minus twice the internal links.
// `fine(b, f, i, j, k, w1, w2, w3, d, m)` gives fine point f = (i, j, k) of block b (m: the
// summed level-0 diagonals it stands for) and returns whether it is active; `act(b, f, i, j, k)`
// only its activity.
// A coarse V point whose diagonal is at or below ncut times its summed level-0 diagonals is a
// near-null mode (a floating conductor collapsed into one aggregate: the constant over it costs
// almost no energy, and the computed diagonal is the cancellation noise of the sums above); it
// leaves the hierarchy (inactive) instead of amplifying its right-hand side by 1 / noise.  The
// conductor-region coarse space carries such modes exactly.
template <typename T, typename Fine, typename Act>
__device__ __forceinline__ void mg_coarsen_point(const MGBlockDesc& fb, const MGBlockDesc& cb, int b, long long t,
                                                 MGLevelDev<T>& C, double ncut, Fine fine, Act act) {
    long long q = t - cb.off;
    int I, J, K;
    mg_ijk(q, cb.n1, cb.n2, I, J, K);
    double d = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0, ms = 0.0;
    bool any = false;
    const long long s2 = fb.n1, s3 = (long long)fb.n1 * fb.n2;
    for (int dk = 0; dk < 2; dk++) for (int dj = 0; dj < 2; dj++) for (int di = 0; di < 2; di++) {
        int i = 2 * I + di, j = 2 * J + dj, k = 2 * K + dk;
        if (i >= fb.n1 || j >= fb.n2 || k >= fb.n3) continue;
        long long f = fb.off + i + (long long)j * s2 + (long long)k * s3;
        T fw1, fw2, fw3, fd, fm;
        if (!fine(b, f, i, j, k, fw1, fw2, fw3, fd, fm)) continue;
        any = true;
        d += fd;
        ms += fm;
        // +x link of f: internal if di == 0, crossing to I+1 if di == 1
        if (i + 1 < fb.n1 && act(b, f + 1, i + 1, j, k)) {
            if (di == 0) d -= 2.0 * fw1;
            else w1 += fw1;
        }
        if (j + 1 < fb.n2 && act(b, f + s2, i, j + 1, k)) {
            if (dj == 0) d -= 2.0 * fw2;
            else w2 += fw2;
        }
        if (k + 1 < fb.n3 && act(b, f + s3, i, j, k + 1)) {
            if (dk == 0) d -= 2.0 * fw3;
            else w3 += fw3;
        }
    }
    C.w1[t] = I + 1 < cb.n1 ? (T)w1 : T(0);
    C.w2[t] = J + 1 < cb.n2 ? (T)w2 : T(0);
    C.w3[t] = K + 1 < cb.n3 ? (T)w3 : T(0);
    C.dg[t] = any ? (T)d : T(1);
    C.mass[t] = any ? (T)ms : T(1);
    const bool null_mode = b == MG_MAX_BLOCKS - 1 && !(d > ncut * ms);
    C.dinv[t] = any && d > 0.0 && !null_mode ? (T)(1.0 / d) : T(0);
}

// level l+1 from the stored arrays of level l
template <typename T>
__global__ void mg_coarsen(MGLevelDev<T> F, MGLevelDev<T> C, double ncut) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= C.total) return;
    const int b = find_block(C, t);
    mg_coarsen_point(F.blk[b], C.blk[b], b, t, C, ncut,
                     [&](int, long long f, int, int, int, T& w1, T& w2, T& w3, T& d, T& m) {
                         w1 = F.w1[f]; w2 = F.w2[f]; w3 = F.w3[f]; d = F.dg[f]; m = F.mass[f];
                         return F.dinv[f] != T(0);
                     },
                     [&](int, long long f, int, int, int) { return F.dinv[f] != T(0); });
}

// level 1 straight from the node coefficients (level 0 keeps no arrays of its own)
template <typename T>
__global__ void mg_coarsen_fine(QGrid g, QCoef<T> c, QStepPar<T> P, T vshift, MGLevelDev<T> F, MGLevelDev<T> C,
                                double ncut) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= C.total) return;
    const int b = find_block(C, t);
    mg_coarsen_point(F.blk[b], C.blk[b], b, t, C, ncut,
                     [&](int bb, long long, int i, int j, int k, T& w1, T& w2, T& w3, T& d, T& m) {
                         const bool a = mg_fine_point(g, c, P, vshift, bb, i + 1, j + 1, k + 1, w1, w2, w3, d);
                         m = d;
                         return a;
                     },
                     [&](int bb, long long, int i, int j, int k) { return mg_fine_active(g, bb, i + 1, j + 1, k + 1); });
}

// a crossing link is only kept if both aggregates are active
template <typename T>
__global__ void mg_mask_links(MGLevelDev<T> C) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= C.total) return;
    const int b = find_block(C, t);
    const MGBlockDesc& cb = C.blk[b];
    long long q = t - cb.off;
    int I, J, K;
    mg_ijk(q, cb.n1, cb.n2, I, J, K);
    if (C.dinv[t] == T(0)) { C.w1[t] = C.w2[t] = C.w3[t] = T(0); return; }
    if (I + 1 < cb.n1 && C.dinv[t + 1] == T(0)) C.w1[t] = T(0);
    if (J + 1 < cb.n2 && C.dinv[t + cb.n1] == T(0)) C.w2[t] = T(0);
    if (K + 1 < cb.n3 && C.dinv[t + (long long)cb.n1 * cb.n2] == T(0)) C.w3[t] = T(0);
}

// A x at point t of block (n1, n2, n3) -- links to inactive points carry w = 0
template <typename T>
__device__ __forceinline__ T apply7(const MGLevelDev<T>& L, const MGBlockDesc& B, long long t, int i, int j, int k,
                                    const T* x) {
    const long long s2 = B.n1, s3 = (long long)B.n1 * B.n2;
    T acc = L.dg[t] * x[t];
    if (i > 0) acc -= L.w1[t - 1] * x[t - 1];
    if (i + 1 < B.n1) acc -= L.w1[t] * x[t + 1];
    if (j > 0) acc -= L.w2[t - s2] * x[t - s2];
    if (j + 1 < B.n2) acc -= L.w2[t] * x[t + s2];
    if (k > 0) acc -= L.w3[t - s3] * x[t - s3];
    if (k + 1 < B.n3) acc -= L.w3[t] * x[t + s3];
    return acc;
}

#define MGC_SWEEPS 8                            // a side: up to this many sweeps have weights of their own
// Weight of sweep s of nu on one side of the cycle: the reciprocal Chebyshev nodes of [0.4, 2], scaled by
// omega / 0.85; one sweep, or more than MGC_SWEEPS: omega.  Their product polynomial is at most 1 / T_3(1.5)
// = 0.11 there for three sweeps; three of weight 0.85 reach 0.34 at 2.  Both sides take the same weights and
// the factors commute, so the cycle stays symmetric.  FGMRES steps a run, equal weights -> these: 96^3 494 ->
// 486, 128^3 336 -> 326, moving plate 256^3 178 -> 167, core 832 -> 800.  Intervals from 0.3, 0.5 and 0.8:
// 256^3 173, 165 and 182, 128^3 326, 328 and 334.
template <typename T>
static inline T mg_weight(T omega, int s, int nu) {
    if (nu < 2 || nu > MGC_SWEEPS) return omega;
    const double a = 0.4, b = 2.0, c = std::cos(3.14159265358979323846 * (2 * s + 1) / (2.0 * nu));
    return (T)((double)omega / 0.85 / (0.5 * (b + a) - 0.5 * (b - a) * c));
}

// ------------------------------------------------------------------ smoother
// Weighted Jacobi on a level of stored links, x' = (1 - omega) x + omega D^-1 (b + sum w x_n); inactive
// points have D^-1 = 0 and stay zero.  Links to points beyond the block's faces are zero, and so are the
// links stored at the last point of a row, a column or a block, which are those "before" the first point
// of the next one: a point needs no (i, j, k), only indexes inside the level's arrays (their values then
// meet a zero link).  All loads of a point are independent, and those of the geometry's links precede the
// wait for the kernel before.  Passes of a level per cycle: 6 instead of 8 (the first two sweeps in one, the
// prolongation with the sweep after it), without index divisions and the diagonal array: 96^3 ellipsoids 168
// -> 163 ms a run, 128^3 209 -> 204, moving plate 256^3 673 -> 647 from one state and 642 -> 643 from another.
template <typename T>
struct MGPoint {
    long long nb[6];                            // neighbours: +1, -1, +n1, -n1, +s3, -s3
    T w[6];
    __device__ __forceinline__ MGPoint(const MGLevelDev<T>& L, const MGBlockDesc& B, long long t) {
        const long long q = t - B.off, n1 = B.n1, s3 = n1 * B.n2;
        const long long d[3] = {1, n1, s3};
        const T* w3[3] = {L.w1, L.w2, L.w3};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            nb[2 * a] = t + d[a] < L.total ? t + d[a] : t;
            nb[2 * a + 1] = q >= d[a] ? t - d[a] : t;
            w[2 * a] = w3[a][t];
            w[2 * a + 1] = q >= d[a] ? w3[a][t - d[a]] : T(0);
        }
    }
};

// one sweep from a zero guess: x = omega D^-1 b
template <typename T>
__global__ void mg_smooth0(MGLevelDev<T> L, const T* b, T omega, T* x) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (t >= L.total) return;
    x[t] = omega * L.dinv[t] * b[t];
}

// the first two sweeps from a zero guess in one pass: x_1 = omega D^-1 b formed at the point and its
// neighbours (a launch and two passes over x less than apart)
template <typename T>
__global__ void __launch_bounds__(256) mg_smooth01(MGLevelDev<T> L, const T* b, T omega1, T omega, T* x) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = t < L.total;
    if (!in) t = 0;
    const MGPoint<T> P(L, L.blk[find_block(L, t)], t);
    T dn[6];
#pragma unroll
    for (int e = 0; e < 6; e++) dn[e] = L.dinv[P.nb[e]];
    const T di = omega * L.dinv[t];
    pdl_wait();
    const T bv = b[t];
    T sum = bv;
#pragma unroll
    for (int e = 0; e < 6; e++) sum += P.w[e] * (omega1 * dn[e] * b[P.nb[e]]);
    if (in) x[t] = (T(1) - omega) * (omega1 * L.dinv[t]) * bv + di * sum;
}

// x_out = x_in + omega D^-1 (b - A x_in)
template <typename T>
__global__ void __launch_bounds__(256) mg_smooth(MGLevelDev<T> L, const T* b, T omega, const T* xin, T* xout) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = t < L.total;
    if (!in) t = 0;
    const MGPoint<T> P(L, L.blk[find_block(L, t)], t);
    const T di = omega * L.dinv[t];
    pdl_wait();
    T sum = b[t];
#pragma unroll
    for (int e = 0; e < 6; e++) sum += P.w[e] * xin[P.nb[e]];
    if (in) xout[t] = (T(1) - omega) * xin[t] + di * sum;
}

// the coarse correction y = x_in + alpha x_c(aggregate) on active points and the first sweep on it in one
// pass (again a launch and two passes over x less): x_out = y + omega D^-1 (b - A y)
template <typename T>
__global__ void __launch_bounds__(256) mg_prolong_smooth(MGLevelDev<T> L, const T* b, T omega, const T* xin, T* xout,
                                                        MGLevelDev<T> C, const T* xc, T alpha) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = t < L.total;
    if (!in) t = 0;
    const int bk = find_block(L, t);
    const MGBlockDesc& fb = L.blk[bk];
    const MGBlockDesc& cb = C.blk[bk];
    const MGPoint<T> P(L, fb, t);
    int i, j, k;
    mg_ijk(t - fb.off, fb.n1, fb.n2, i, j, k);
    const int c2 = cb.n1, c3 = cb.n1 * cb.n2;
    const T* x0 = xc + cb.off;
    const int I = i >> 1, J = (j >> 1) * c2, K = (k >> 1) * c3;
    // the aggregates of the point and of its neighbours (inside the block; a neighbour beyond it has no link)
    const int c[7] = {I + J + K,
                      (min(i + 1, fb.n1 - 1) >> 1) + J + K, (max(i - 1, 0) >> 1) + J + K,
                      I + (min(j + 1, fb.n2 - 1) >> 1) * c2 + K, I + (max(j - 1, 0) >> 1) * c2 + K,
                      I + J + (min(k + 1, fb.n3 - 1) >> 1) * c3, I + J + (max(k - 1, 0) >> 1) * c3};
    const T di = omega * L.dinv[t];
    pdl_wait();
    T sum = b[t];
#pragma unroll
    for (int e = 0; e < 6; e++) sum += P.w[e] * (xin[P.nb[e]] + alpha * x0[c[e + 1]]);
    if (in) xout[t] = di != T(0) ? (T(1) - omega) * (xin[t] + alpha * x0[c[0]]) + di * sum : T(0);
}

// residual of the fine level summed over each aggregate -> coarse right-hand side.  A thread per fine
// point (tiles of 32 x 4 x 2 points, even origins), the eight residuals of an aggregate added through a
// shuffle and shared memory: a thread per coarse point left a chain of eight 7-point rows (10-16 us a
// launch on levels of 25^3 to 129^3 points; 65^3: 11 us then, 7 us now).
#define MGR_X 32
#define MGR_Y 4
#define MGR_Z 2
template <typename T>
__global__ void __launch_bounds__(MGR_X * MGR_Y * MGR_Z) mg_restrict(MGLevelDev<T> F, const T* bf, const T* xf,
                                                                    MGLevelDev<T> C, T* bc, int xtiles) {
    __shared__ T sh[MGR_Z][MGR_Y][MGR_X];
    const int b = blockIdx.x / xtiles;
    const MGBlockDesc& fb = F.blk[b];
    const MGBlockDesc& cb = C.blk[b];
    const int i = (blockIdx.x - b * xtiles) * MGR_X + threadIdx.x, j = blockIdx.y * MGR_Y + threadIdx.y;
    const int k = blockIdx.z * MGR_Z + threadIdx.z;
    T r = T(0);
    pdl_wait();
    if (i < fb.n1 && j < fb.n2 && k < fb.n3) {
        const long long f = fb.off + i + (long long)j * fb.n1 + (long long)k * fb.n1 * fb.n2;
        if (F.dinv[f] != T(0)) r = bf[f] - apply7(F, fb, f, i, j, k, xf);
    }
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    sh[threadIdx.z][threadIdx.y][threadIdx.x] = r;
    __syncthreads();
    if (threadIdx.z != 0 || ((threadIdx.x | threadIdx.y) & 1)) return;
    const int I = i >> 1, J = j >> 1, K = k >> 1;
    if (I >= cb.n1 || J >= cb.n2 || K >= cb.n3) return;
    r = (sh[0][threadIdx.y][threadIdx.x] + sh[0][threadIdx.y + 1][threadIdx.x]) +
        (sh[1][threadIdx.y][threadIdx.x] + sh[1][threadIdx.y + 1][threadIdx.x]);
    bc[cb.off + I + (long long)J * cb.n1 + (long long)K * cb.n1 * cb.n2] = r;
}

// ------------------------------------------------------------------ coarse sub-cycle
// The last levels of a cycle in one launch: one cluster of CTAs (16, or 8 where the chip cannot place 16)
// per block runs their whole V-cycle for that block.  A level's planes are dealt out to the CTAs in slabs (a level of at most
// MGC_LOCAL points is the first CTA's alone); links, right-hand side and x live in shared memory, x
// with a halo plane on each side, the boundary planes are written to the neighbours' halos through
// distributed shared memory, and a pass ends with a cluster barrier.
// These levels are bound by latency, not by bytes (33^3 points of a block are 0.1 MB per array): a
// launch per sweep cost 2.8-4 us each, and the smallest levels in one CTA with their data in L2 20-36 us.
// So the links are copied to shared memory once per cycle (the lower levels' while the first one runs);
// the passes are short loops that every level shares (unrolled by the points of a thread, with the links
// in registers, a level's first pass waited for its instructions: 15,000 clocks for a sweep of 4,000);
// and levels whose cluster barriers (600 clocks) would outweigh their work stay in one CTA.
// Per cycle on the A blocks, levels 25^3 to 4^3: 63 us as nine launches before, 24 us now; 33^3 to 5^3:
// 76 us as seventeen, 36 us now.  Measured and not taken: 8 CTAs (3 % slower on the runs), 1024 or 256
// threads (7 %, 2-5 %), one-CTA levels of up to 2500 points (3 %).
#define MGC_THREADS 512
#define MGC_LEVELS 8
#define MGC_LOCAL 1024
#define MGC_SMEM (216 * 1024)
template <typename T>
struct MGSub {
    int nl;                                     // levels; the last is the coarsest
    int lg;                                     // 2^lg CTAs in the cluster
    T w1[MGC_SWEEPS], w2[MGC_SWEEPS];           // weights of the sweeps before and after the correction
    MGLevelDev<T> L[MGC_LEVELS];
};
// planes of a level that one CTA of 2^lg holds, and the shared memory (elements) of a level: two copies of x
// with halo planes and an element on either side, the right-hand side, and (not the last level) dinv,
// w1, w2, w3 with the plane before
__host__ __device__ __forceinline__ int mgc_planes(const MGBlockDesc& B, int lg) {
    return (long long)B.n1 * B.n2 * B.n3 <= MGC_LOCAL ? B.n3 : (B.n3 + (1 << lg) - 1) >> lg;
}
__host__ __device__ __forceinline__ long long mgc_xlen(const MGBlockDesc& B, int lg) {
    return (long long)(mgc_planes(B, lg) + 2) * B.n1 * B.n2 + 2;
}
__host__ __device__ __forceinline__ long long mgc_len(const MGBlockDesc& B, int lg, bool links) {
    const int P = mgc_planes(B, lg);
    return 2 * mgc_xlen(B, lg) + (long long)(P + (links ? 4 * (P + 1) : 0)) * B.n1 * B.n2;
}
extern __shared__ __align__(16) unsigned char mgc_raw[];

// one CTA's slab of a level; x, b, w: indexes in the CTA's shared memory (of T): own point q of x at
// x + which * xlen + s3 + q, its dinv and links at w + s3 + q + (0..3) * P4
struct MGSlab {
    int n1, n2, n3, s3, P, P3, P4, z0, np, rank;    // P: planes of a full slab, np: points of this one
    int x, xlen, b, w;
    bool dn, up, spread;                        // a neighbour holds the plane before / after; more than one CTA
    __device__ __forceinline__ MGSlab(const MGBlockDesc& B, int lg, int c, int at) {
        n1 = B.n1;
        n2 = B.n2;
        n3 = B.n3;
        s3 = B.n1 * B.n2;
        P = mgc_planes(B, lg);
        P3 = P * s3;
        P4 = P3 + s3;
        rank = c;
        z0 = min(c * P, B.n3);
        np = (min(z0 + P, B.n3) - z0) * s3;
        dn = c > 0 && np > 0;
        up = z0 + P < B.n3;
        spread = P < B.n3;
        x = at + 1;
        xlen = (int)mgc_xlen(B, lg);
        b = at + 2 * xlen;
        w = b + P3;
    }
};

template <typename T>
struct MGCluster {
    cg::cluster_group cl;
    T* sm;                                      // mgc_raw's part of T, the same place in every CTA
    __device__ __forceinline__ void sync(bool all) {
        if (all) cl.sync();
        else __syncthreads();
    }
    __device__ __forceinline__ T* remote(int at, int rank) { return cl.map_shared_rank(sm + at, rank); }
    // a value of the slab, and into the neighbours' halos from its outer planes
    __device__ __forceinline__ void put(const MGSlab& S, int x, int q, T v) {
        sm[x + S.s3 + q] = v;
        if (S.dn && q < S.s3) *remote(x + S.s3 + S.P3 + q, S.rank - 1) = v;
        if (S.up && q >= S.np - S.s3) *remote(x + (q - (S.np - S.s3)), S.rank + 1) = v;
    }
    // b + sum w x_n at own point q.  The links of the last point of a row, a column or the block are
    // zero, so the ones "before" the first point are too (zeros in the plane before the block).
    __device__ __forceinline__ T rest(const MGSlab& S, int x, int q) const {
        const T* y = sm + x + S.s3 + q;
        const T* w = sm + S.w + S.s3 + q;
        return sm[S.b + q] + w[S.P4] * y[1] + w[S.P4 - 1] * y[-1] + w[2 * S.P4] * y[S.n1] +
               w[2 * S.P4 - S.n1] * y[-S.n1] + w[3 * S.P4] * y[S.s3] + w[3 * S.P4 - S.s3] * y[-S.s3];
    }
    // x' = (1 - omega) x + omega D^-1 (b + sum w x_n) from copy cur into the other
    __device__ __forceinline__ void sweep(const MGSlab& S, int& cur, T omega) {
        const int x = S.x + cur * S.xlen;
        cur ^= 1;
#pragma unroll 2
        for (int q = threadIdx.x; q < S.np; q += MGC_THREADS)
            put(S, S.x + cur * S.xlen, q, (T(1) - omega) * sm[x + S.s3 + q] + omega * sm[S.w + S.s3 + q] * rest(S, x, q));
        sync(S.spread);
    }
};

template <typename T>
__global__ void __launch_bounds__(MGC_THREADS, 1) mg_sub(const __grid_constant__ MGSub<T> sub,
                                                       const double* __restrict__ minv,
                                                       const long long* __restrict__ moff, T alpha, int nu1,
                                                       int nu2) {
    const int lg = sub.lg, size = 1 << lg, b = blockIdx.x >> lg, last = sub.nl - 1, tid = threadIdx.x;
    const int m = sub.L[last].blk[b].n1 * sub.L[last].blk[b].n2 * sub.L[last].blk[b].n3;
    double* db = reinterpret_cast<double*>(mgc_raw);
    MGCluster<T> G{cg::this_cluster(), reinterpret_cast<T*>(mgc_raw) + m * (int)(sizeof(double) / sizeof(T))};
    const int c = (int)G.cl.block_rank();
    __shared__ int at[MGC_LEVELS + 1];
    if (tid == 0) {
        int o = 0;
        for (int l = 0; l <= last; l++) { at[l] = o; o += (int)mgc_len(sub.L[l].blk[b], lg, l < last); }
    }
    __syncthreads();
    auto slab = [&](int l) { return MGSlab(sub.L[l].blk[b], lg, c, at[l]); };
    // the links of every level on their way; x's copies start at
    // zero: the halos beyond the grid are never written, zero like the links that point there
#pragma unroll 1
    for (int l = 0; l <= last; l++) {
        const MGSlab S = slab(l);
        if (l < last && S.np > 0) {
            const MGLevelDev<T>& L = sub.L[l];
            const long long first = L.blk[b].off + (long long)(S.z0 - 1) * S.s3;
#pragma unroll 1
            for (int q = tid; q < S.np + S.s3; q += MGC_THREADS) {
                const bool in = S.z0 > 0 || q >= S.s3;
                const long long t = in ? first + q : L.blk[b].off;
                T* d = G.sm + S.w + q;
                cp_async_elem(d, L.dinv + t, in);
                cp_async_elem(d + S.P4, L.w1 + t, in);
                cp_async_elem(d + 2 * S.P4, L.w2 + t, in);
                cp_async_elem(d + 3 * S.P4, L.w3 + t, in);
            }
        }
        if (l == 0) cp_async_commit();
    }
    cp_async_commit();
#pragma unroll 1
    for (int l = 0; l <= last; l++)
        for (int q = tid; q < 2 * (int)mgc_xlen(sub.L[l].blk[b], lg); q += MGC_THREADS) G.sm[at[l] + q] = T(0);
    // this warp's first row of the coarsest inverse: its loads are out of the way when the row is needed
    const double* M = minv + moff[b];
    const int lane = tid & 31, r0 = c * (MGC_THREADS / 32) + (tid >> 5);
    double mrow[4];
#pragma unroll
    for (int e = 0; e < 4; e++) mrow[e] = r0 < m && lane + 32 * e < m ? M[(long long)r0 * m + lane + 32 * e] : 0.0;
    // the links are the geometry's; the first level's right-hand side is the kernel's before this one
    pdl_wait();
    if (last > 0) {
        const MGSlab S = slab(0);
        const long long off = sub.L[0].blk[b].off + (long long)S.z0 * S.s3;
        for (int q = tid; q < S.np; q += MGC_THREADS) G.sm[S.b + q] = sub.L[0].b[off + q];
    }
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    G.cl.sync();
    // down: pre-smoothing from zero, and the residual summed over each 2x2x2 aggregate into the
    // right-hand side of the CTA that holds the coarse point
#pragma unroll 1
    for (int l = 0; l < last; l++) {
        if (l == 1) {                            // the copies of every thread
            cp_async_wait_all();
            __syncthreads();
        }
        const MGSlab S = slab(l), SC = slab(l + 1);
        if (!S.spread && c != 0) break;
#pragma unroll 2
        for (int q = tid; q < S.np; q += MGC_THREADS) G.put(S, S.x, q, sub.w1[0] * G.sm[S.w + S.s3 + q] * G.sm[S.b + q]);
        G.sync(S.spread);
        int cur = 0;
#pragma unroll 1
        for (int s = 1; s < nu1; s++) G.sweep(S, cur, sub.w1[s & (MGC_SWEEPS - 1)]);
        const int X = S.x + cur * S.xlen, R = S.x + (cur ^ 1) * S.xlen;   // the residual into the other copy
#pragma unroll 2
        for (int q = tid; q < S.np; q += MGC_THREADS) {
            const T di = G.sm[S.w + S.s3 + q];
            G.put(S, R, q, di != T(0) ? G.rest(S, X, q) - G.sm[X + S.s3 + q] / di : T(0));
        }
        G.sync(S.spread);
        const int n1 = S.n1, s3 = S.s3;
        const int K0 = (S.z0 + 1) >> 1, K1 = (S.z0 + S.np / s3 + 1) >> 1;   // coarse planes whose first fine plane is here
#pragma unroll 1
        for (int q = tid; q < (K1 - K0) * SC.s3; q += MGC_THREADS) {
            int I, J, K;
            mg_ijk(q, SC.n1, SC.n2, I, J, K);
            K += K0;
            const T* r = G.sm + R + s3 + (2 * K - S.z0) * s3 + 2 * J * n1 + 2 * I;
            const bool i2 = 2 * I + 1 < S.n1, j2 = 2 * J + 1 < S.n2, k2 = 2 * K + 1 < S.n3;
            T a = r[0];
            if (i2) a += r[1];
            if (j2) a += r[n1];
            if (i2 && j2) a += r[n1 + 1];
            if (k2) {
                a += r[s3];
                if (i2) a += r[s3 + 1];
                if (j2) a += r[s3 + n1];
                if (i2 && j2) a += r[s3 + n1 + 1];
            }
            const int owner = K / SC.P;
            *G.remote(SC.b + (K - owner * SC.P) * SC.s3 + J * SC.n1 + I, owner) = a;
        }
        G.sync(S.spread);
    }
    cp_async_wait_all();
    G.cl.sync();
    {   // coarsest: x = Minv b (FP64 dense; pseudo-inverse for V), b and x in the first CTA, a warp per row
        // over the cluster: one SM's FP64 rate (2 FMA per clock) would take 4 us for 125 rows
        const MGSlab S = slab(last);
        const long long off = sub.L[last].blk[b].off;
        const T* rb = G.remote(S.b, 0);
        for (int q = tid; q < m; q += MGC_THREADS) db[q] = (double)(last == 0 ? sub.L[0].b[off + q] : rb[q]);
        __syncthreads();
        T* rx = last == 0 ? sub.L[0].x + off : G.remote(S.x + S.s3, 0);
#pragma unroll 1
        for (int r = r0; r < m; r += size * (MGC_THREADS / 32)) {
            double acc = 0.0;
            int q = lane;
            if (r == r0) {
#pragma unroll
                for (int e = 0; e < 4; e++, q += 32) acc += mrow[e] * (q < m ? db[q] : 0.0);
            }
#pragma unroll 1
            for (; q < m; q += 32) acc += M[(long long)r * m + q] * db[q];
            acc = qWarpSum(acc);
            if (lane == 0) rx[r] = (T)acc;
        }
        G.cl.sync();
    }
    // up: the coarse correction and the post-smoothing.  Where the last sweep of a level left x: the copy
    // alternates with every sweep after the first
    const int down = (nu1 - 1) & 1, done = (nu1 - 1 + nu2) & 1;
#pragma unroll 1
    for (int l = last - 1; l >= 0; l--) {
        const MGSlab S = slab(l), SC = slab(l + 1);
        if (!S.spread && c != 0) continue;
        if (S.spread && !SC.spread && l + 1 < last) G.cl.sync();   // the first CTA has the coarse correction
        const int X = S.x + down * S.xlen, XC = SC.x + (l + 1 == last ? 0 : done * SC.xlen) + SC.s3;
#pragma unroll 2
        for (int q = tid; q < S.np; q += MGC_THREADS) {
            int i, j, k;
            mg_ijk(q, S.n1, S.n2, i, j, k);
            const int K = (S.z0 + k) >> 1, owner = K / SC.P;
            const T xc = *G.remote(XC + (K - owner * SC.P) * SC.s3 + (j >> 1) * SC.n1 + (i >> 1), owner);
            G.put(S, X, q, G.sm[S.w + S.s3 + q] != T(0) ? G.sm[X + S.s3 + q] + alpha * xc : T(0));
        }
        G.sync(S.spread);
        int cur = down;
#pragma unroll 1
        for (int s = 0; s < nu2; s++) G.sweep(S, cur, sub.w2[s & (MGC_SWEEPS - 1)]);
    }
    if (last > 0) {
        const MGSlab S = slab(0);
        const int x = S.x + done * S.xlen + S.s3;
        const long long off = sub.L[0].blk[b].off + (long long)S.z0 * S.s3;
        for (int q = tid; q < S.np; q += MGC_THREADS) sub.L[0].x[off + q] = G.sm[x + q];
    }
}

// ---------------------------------------------------------------------------
// Level-0 kernels on node tiles.  Level 0 of every block is the global unknown
// vector itself, and its 7-point operators are the self couplings of the rows
// of qms_operator.cu, so they read the same staged node coefficients instead
// of stored per-point links:
//   KIND 0: x = omega D^-1 b                      (first sweep, zero guess)
//   KIND 1: x_out = x_in + omega D^-1 (b - A x_in)
//   KIND 3: the first two sweeps from a zero guess in one pass (scaled b only): the
//           first sweep is x_1 = omega isc b pointwise (the diagonal cancels against
//           the row scaling), so b's tile is staged in x_in's place and scaled on use
//   KIND 2: b_c = sum over each 2x2x2 aggregate of (b - A x_in)  (restriction
//           fused with the residual; no atomics, fixed order)
// b is scaled pointwise by the row scaling of the outer system when bscale is
// given; that scaling is the operator diagonal, formed here from the coefficients.
// A stage of a march is x's plane k + 1 (all components, +-1 halo in i and j) and
// the coefficients' plane k, two TMA copies on one mbarrier, issued two planes
// ahead; b is fetched into registers one plane ahead.
// The kernels were bound by instruction issue, not by bytes, so: on grids of 1216 tiles or more a thread has
// two rows (ROWS; j and j + 1: their common coefficients and x are read once, address arithmetic and
// the plane's barrier shared), on smaller ones, where the march's latency counts, one; what plane k - 1
// contributes (x and three coefficients at the thread's own node) stays in
// registers; the sweeps use x' = (1 - omega) x + omega D^-1 (b + sum w x_n) (the
// restriction keeps the difference form, whose rounding scales with the variation
// of x); on cubic cells (UNI) the links are the coefficients themselves, the factor
// 1/h^2 left out where it cancels; the Dirichlet tests are split into a per-thread
// (i, j) part and a per-plane k part, and Dirichlet points, zero in every vector
// here, are not written; D^-1 is a fast reciprocal in FP32 (a preconditioner needs
// no correctly rounded divide).
// Before these (coefficients and x of three planes read from shared memory, links multiplied by 1/h^2,
// two mbarriers per plane, one plane ahead), ms per run of steps: 96^3 202 -> 191, 128^3 244 -> 229,
// moving plate 256^3 780 -> 717, 64^3 in FP64 411 -> 337.  Two rows per thread instead of one: 96^3 191 ->
// 186, 128^3 228 -> 219, 256^3 717 -> 690, but 48^3 161 -> 169 and FP64 as before (one row there).
// The A blocks' sweep at 192^3: 94.7 us and 87.7 M warp instructions before, 67.8 us and 47.1 M now, with issue
// 62 % active and DRAM at 64 %: latency (staged planes, the plane's barrier) is what is left.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T mg_rcp(T d) {
    if constexpr (sizeof(T) == 4) return __fdividef(1.0f, d);
    else return T(1) / d;
}

// QS selects the blocks a cycle works on: 0 all four, 1 the three A blocks, 2 the V block
// (then only the three conductivities are staged).  xmap / cmap cover exactly those blocks /
// arrays; b, xout and the rows stay those of the whole padded vector, bc that of the level-1
// view of the same blocks.
template <int QS> struct MG0Set {
    static constexpr int NQ = QS == 0 ? 4 : (QS == 1 ? 3 : 1), Q0 = QS == 2 ? 3 : 0;
    static constexpr int NC = QS == 2 ? 3 : 6, C0 = QS == 2 ? 3 : 0;
    static constexpr bool A = QS != 2, V = QS != 1;
};

// Coefficient tiles of the level-0 kernels: bf16 in an FP32 hierarchy (a preconditioner needs
// no more than its ~3 significant digits, and the six node coefficients are 40 % of a sweep's
// DRAM traffic in FP32), the hierarchy's own type in FP64.
template <typename T> struct MG0Coef { using type = T; };
template <> struct MG0Coef<float> { using type = __nv_bfloat16; };
__device__ __forceinline__ float mg_cf(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ double mg_cf(double v) { return v; }

template <typename T, int KIND, int QS, bool UNI, int ROWS>
__global__ void __launch_bounds__(OTX * OTY / ROWS, sizeof(T) == 4 ? (ROWS == 1 ? QMS_STENCIL_MINB : 6) : 2)
mg0_tiled(QGrid g, QStepPar<T> P, T vshift, T omega, T omega1, const T* b, int scaled,
          const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap cmap, T* xout,
          MGLevelDev<T> C, T* bc, unsigned* err) {
    using S = MG0Set<QS>;
    using CT = typename MG0Coef<T>::type;
    using TL = PLTiles<T, S::NQ, S::NC, CT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* xsm = reinterpret_cast<T*>(smem_raw);                  // [4 slots][NQ][PLXY][PLX]
    CT* csm = reinterpret_cast<CT*>(smem_raw + 4 * TL::XSLOT * sizeof(T));   // [3 slots][NC][PLCY][CX]
    __shared__ __align__(8) uint64_t bar[4], pbar;
    __shared__ T red[KIND == 2 && ROWS == 1 ? S::NQ : 1][OTY][OTX];
    constexpr bool STAGE = KIND != 0;
    constexpr int NQ = S::NQ, Q0 = S::Q0, R = ROWS;
    const int tid = threadIdx.x + OTX * threadIdx.y;
    const int i0 = blockIdx.x * OTX + 1, j0 = blockIdx.y * OTY + 1, k0 = blockIdx.z * g.okb + 1;
    // this thread's nodes: (i, j + r), r < R
    const int li = threadIdx.x + 1, lj = threadIdx.y * R + 1;
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y * R;
    const int kend = min(k0 + g.okb - 1, g.Nz);
    const QPL L = qms_pl(g);
    const int cx = i0 - 1, cy = j0 - 2;
    auto load_x = [&](int kk, uint64_t* on) { tma_load_4d(xsm + (kk & 3) * TL::XSLOT, &xmap, cx, cy, kk - 1, 0, on); };
    auto load_c = [&](int kk, uint64_t* on) { tma_load_4d(csm + (kk % 3) * TL::CSLOT, &cmap, cx, cy, kk - 1, 0, on); };
    // what plane k needs beyond the planes before it: x's plane k + 1 and the coefficients' plane k
    auto issue = [&](int k) {
        uint64_t* on = &bar[(k - k0) & 3];
        mbar_expect_tx(on, (STAGE ? TL::XBYTES : 0u) + TL::CBYTES);
        if (STAGE) load_x(k + 1, on);
        load_c(k, on);
    };
    if (tid == 0) {
        for (int q = 0; q < 4; q++) mbar_init(&bar[q], 1);
        mbar_init(&pbar, 1);
        fence_mbar_init();
        mbar_expect_tx(&pbar, (STAGE ? 2 * TL::XBYTES : 0u) + TL::CBYTES);
        load_c(k0 - 1, &pbar);                  // (the coefficients are the geometry's)
        pdl_wait();
        if (STAGE) {
            load_x(k0 - 1, &pbar);
            load_x(k0, &pbar);
        }
        issue(k0);
        if (k0 + 1 <= kend) issue(k0 + 1);
    } else {
        pdl_wait();
    }
    __syncthreads();
    bool ok = mbar_wait(&pbar, 0, err);
    // the rows this thread solves: inside the grid and no Dirichlet row but for its k terms
    const bool fxA = i <= 2 || i >= g.Nx - 1;
    bool in[R], act[4][R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int jr = j + r;
        const bool fyA = jr <= 2 || jr >= g.Ny - 1;
        in[r] = i <= g.Nx && jr <= g.Ny;
        act[0][r] = in[r] && !(fyA || i == 1 || i >= g.xs);
        act[1][r] = in[r] && !(fxA || jr == 1 || jr >= g.ys);
        act[2][r] = in[r] && !(fxA || fyA);
        act[3][r] = act[2][r];
    }
    // offset of node (i, j) at plane k in a block (32-bit: checked at creation); block q's row r is
    // q * comp + nd + r * P
    const int comp = (int)L.comp, plane = g.Ny * L.P, pitch = L.P;
    int nd = ((k0 - 1) * g.Ny + (j - 1)) * L.P + i;
    const T iscV = scaled ? T(1) / (T(1) + vshift) : T(1);
    // 1/h^2 of the links, and the mass and b in their units
    const T wx = UNI ? T(1) : P.idx2, wy = UNI ? T(1) : P.idy2, wz = UNI ? T(1) : P.idz2;
    const T unit = UNI ? P.idx2 : T(1), iunit = UNI ? T(1) / P.idx2 : T(1), wm = P.idt * iunit;
    T acc[4] = {T(0), T(0), T(0), T(0)};
    // right-hand side of this thread's rows, fetched one plane ahead so that the loads are in flight
    // while the previous plane is computed (KIND 3 has it in its tiles).  The row scaling of the outer
    // system is the operator's diagonal, which is this level's diagonal d divided by dscale (1 + vshift
    // on V, 1 on A): it is formed from the staged coefficients, not read.
    T bn[4][R];
    auto fetch_b = [&](int kk, int n) {
#pragma unroll
        for (int q = Q0; q < Q0 + NQ; q++)
#pragma unroll
            for (int r = 0; r < R; r++)
                bn[q][r] = KIND != 3 && act[q][r] && (q != 2 || kk <= g.zs) ? b[q * comp + n + r * pitch] : T(0);
    };
    fetch_b(k0, nd);
#define CF(s, q, dj, di) ((T)mg_cf((s)[((q) - S::C0) * PLCY * TL::CX + (lj + (dj)) * TL::CX + li + (di)]))
#define XS(s, q, dj, di) (s)[((q) - Q0) * PLXY * PLX + (lj + (dj)) * PLX + li + (di)]
    // plane k - 1 at these nodes: x of every component and the coefficients of the links along k
    T xm[4][R], xc[4][R], cm[6][R];
    {
        const T* p0 = xsm + ((k0 - 1) & 3) * TL::XSLOT;
        const T* p1 = xsm + (k0 & 3) * TL::XSLOT;
        const CT* cp = csm + ((k0 - 1) % 3) * TL::CSLOT;
#pragma unroll
        for (int r = 0; r < R; r++) {
#pragma unroll
            for (int q = Q0; q < Q0 + NQ; q++) {
                xm[q][r] = STAGE && ok ? XS(p0, q, r, 0) : T(0);
                xc[q][r] = STAGE && ok ? XS(p1, q, r, 0) : T(0);
            }
            if (S::A)
#pragma unroll
                for (int q = 0; q < 3; q++) cm[q][r] = ok ? CF(cp, q, r, 0) : T(0);
            if (S::V) cm[5][r] = ok ? CF(cp, 5, r, 0) : T(0);
        }
    }
    for (int k = k0; k <= kend; k++) {
        T bv[4][R];
#pragma unroll
        for (int q = Q0; q < Q0 + NQ; q++)
#pragma unroll
            for (int r = 0; r < R; r++) bv[q][r] = bn[q][r];
        if (k < kend) fetch_b(k + 1, nd + plane);
        if (!__syncthreads_and(ok)) break;         // plane k-1's slots free; uniform stop on a lost copy
        if (tid == 0 && k + 2 <= kend) {
            fence_proxy_async();
            issue(k + 2);
        }
        ok = mbar_wait(&bar[(k - k0) & 3], (unsigned)(((k - k0) >> 2) & 1), err);
        const T* x0 = xsm + (k & 3) * TL::XSLOT;
        const T* xq = xsm + ((k + 1) & 3) * TL::XSLOT;
        const CT* cc = csm + (k % 3) * TL::CSLOT;
        const bool kA = k > 2 && k < g.Nz - 1;          // k terms of qFixX / qFixY / qFixV
        const bool kZ = k > 1 && k < g.zs;              // k term of qFixZ
        T res[4];                                       // KIND 2: this plane's residual, summed over the rows
        // one component: links along x (cxp at the node, cxm before it), along y (ypr: row r, ym0: before
        // row 0) and along z (zpr, zmr), extra diagonal
        auto point = [&](int q, bool kok, const T (&cxp)[R], const T (&cxm)[R], const T (&cyp)[R], T cym,
                         const T (&czp)[R], const T (&czm)[R], const T (&mass)[R], T dscale, T isc) {
            T xp[R];
            res[q] = T(0);
#pragma unroll
            for (int r = 0; r < R; r++) xp[r] = STAGE ? XS(xq, q, r, 0) : T(0);
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (!(kok && act[q][r])) continue;
                const T wxp = cxp[r] * wx, wxm = cxm[r] * wx, wyp = cyp[r] * wy, wym = (r > 0 ? cyp[r > 0 ? r - 1 : 0] : cym) * wy;
                const T wzp = czp[r] * wz, wzm = czm[r] * wz;
                const T wsum = ((wxp + wxm) + (wyp + wym)) + (wzp + wzm);
                const T d = (wsum + mass[r]) * dscale;
                const int row = q * comp + nd + r * pitch;
                const T xs = xc[q][r];
                if (KIND == 0) {
                    xout[row] = scaled ? omega * isc * bv[q][r] : omega * bv[q][r] * iunit * mg_rcp(d);
                    continue;
                }
                const T xip = XS(x0, q, r, 1), xim = XS(x0, q, r, -1);
                const T xjp = r + 1 < R ? xc[q][r + 1 < R ? r + 1 : r] : XS(x0, q, R, 0);
                const T xjm = r > 0 ? xc[q][r > 0 ? r - 1 : 0] : XS(x0, q, -1, 0);
                if (KIND == 2) {
                    // difference form: d - sum(w) is the mass term, or the diagonal shift of V
                    const T Ax = wxp * (xs - xip) + wxm * (xs - xim) + wyp * (xs - xjp) + wym * (xs - xjm) +
                                 wzp * (xs - xp[r]) + wzm * (xs - xm[q][r]) + (d - wsum) * xs;
                    res[q] += scaled ? unit * (bv[q][r] * d * isc - Ax) : bv[q][r] - unit * Ax;
                } else {
                    const T nb = wxp * xip + wxm * xim + wyp * xjp + wym * xjm + wzp * xp[r] + wzm * xm[q][r];
                    // KIND 3: the staged values are b; x_1 = c b with c = omega1 isc, and the neighbours' sum
                    // scales with it (omega1: the first sweep's weight, omega: the second's)
                    if (KIND == 3) {
                        const T cq = omega1 * isc;
                        xout[row] = ((T(1) - omega) * cq + omega * isc) * xs + omega * cq * (nb * mg_rcp(d));
                    } else if (scaled) {
                        xout[row] = (T(1) - omega) * xs + omega * (isc * bv[q][r] + nb * mg_rcp(d));
                    } else {
                        xout[row] = (T(1) - omega) * xs + omega * (iunit * bv[q][r] + nb) * mg_rcp(d);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                xm[q][r] = xc[q][r];
                xc[q][r] = xp[r];
            }
        };
        if constexpr (S::A) {
            T c[3][R], ci[3][R], cj[3], mass[R];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                cj[q] = CF(cc, q, -1, 0);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    c[q][r] = CF(cc, q, r, 0);
                    ci[q][r] = CF(cc, q, r, -1);
                }
            }
#pragma unroll
            for (int r = 0; r < R; r++) mass[r] = CF(cc, 3, r, 0) * wm;
            point(0, kA, c[0], ci[0], c[2], cj[2], c[1], cm[1], mass, T(1), T(1));
#pragma unroll
            for (int r = 0; r < R; r++) mass[r] = CF(cc, 4, r, 0) * wm;
            point(1, kA, c[2], ci[2], c[1], cj[1], c[0], cm[0], mass, T(1), T(1));
#pragma unroll
            for (int r = 0; r < R; r++) mass[r] = CF(cc, 5, r, 0) * wm;
            point(2, kZ, c[1], ci[1], c[0], cj[0], c[2], cm[2], mass, T(1), T(1));
#pragma unroll
            for (int q = 0; q < 3; q++)
#pragma unroll
                for (int r = 0; r < R; r++) cm[q][r] = c[q][r];
        }
        if constexpr (S::V) {
            const T fl = P.sigfloor;
            T s0[R], s0i[R], s1[R], s2[R], s2m[R], none[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                s0[r] = fmax(CF(cc, 3, r, 0), fl);
                s0i[r] = fmax(CF(cc, 3, r, -1), fl);
                s1[r] = fmax(CF(cc, 4, r, 0), fl);
                s2[r] = fmax(CF(cc, 5, r, 0), fl);
                s2m[r] = fmax(cm[5][r], fl);
                none[r] = T(0);
            }
            point(3, kA, s0, s0i, s1, fmax(CF(cc, 4, -1, 0), fl), s2, s2m, none, T(1) + vshift, iscV);
#pragma unroll
            for (int r = 0; r < R; r++) {
                cm[5][r] = s2[r];
            }
        }
        nd += plane;
        if (KIND == 2) {
            // aggregates: i pairs (2p+1, 2p+2) a shuffle, j pairs this thread's two rows or, with one row per
            // thread, shared memory, k pairs (odd, even) registers
            const bool first = ((k - k0) & 1) == 0;
            T v[4];
#pragma unroll
            for (int q = Q0; q < Q0 + NQ; q++) v[q] = res[q] + __shfl_xor_sync(0xffffffffu, res[q], 1);
            if constexpr (R == 1) {
#pragma unroll
                for (int q = 0; q < NQ; q++) red[q][threadIdx.y][threadIdx.x] = v[q + Q0];
                __syncthreads();
#pragma unroll
                for (int q = 0; q < NQ; q++) v[q + Q0] += red[q][threadIdx.y ^ 1][threadIdx.x];
            }
#pragma unroll
            for (int q = Q0; q < Q0 + NQ; q++) acc[q] = first ? v[q] : acc[q] + v[q];
            if (!(threadIdx.x & 1) && (R > 1 || !(threadIdx.y & 1)) && (!first || k == kend)) {
                const int I = (i - 1) >> 1, J = (j - 1) >> 1, K = (k - 1) >> 1;
#pragma unroll
                for (int q = Q0; q < Q0 + NQ; q++) {
                    const MGBlockDesc& cb = C.blk[q - Q0];
                    if (I < cb.n1 && J < cb.n2 && K < cb.n3)
                        bc[cb.off + I + (long long)J * cb.n1 + (long long)K * cb.n1 * cb.n2] =
                            acc[q];
                }
            }
        }
    }
#undef CF
#undef XS
}

// level 0: x += alpha P x_c on the active points (the Dirichlet points of every component stay zero; C and xc: the level-1 view of the blocks of QS).  A thread has one 16-byte packet of
// columns (columns W v .. W v + W - 1 are i = W v ..; pairs (2I + 1, 2I + 2) share a coarse value) of each
// component: bound by the bytes of x, which a thread per node moved 4 at a time (256^3, the A blocks:
// 147 us before; runs of steps 128^3 220 -> 214 ms, 256^3 713 -> 694).
#define MGP_X 16
#define MGP_Y 16
template <typename T, int QS>
__global__ void __launch_bounds__(MGP_X * MGP_Y) mg0_prolong(QGrid g, T* x, MGLevelDev<T> C, const T* xc,
                                                            T alpha) {
    using S = MG0Set<QS>;
    constexpr int W = 16 / (int)sizeof(T);
    struct alignas(16) Packet { T v[W]; };
    const QPL L = qms_pl(g);
    const int c0 = (blockIdx.x * MGP_X + threadIdx.x) * W, j = blockIdx.y * MGP_Y + threadIdx.y + 1, k = blockIdx.z + 1;
    pdl_wait();
    if (c0 >= g.xs || j > g.ys) return;                       // i >= xs, j > ys: Dirichlet rows only
    const int J = (j - 1) >> 1, K = (k - 1) >> 1, I0 = (c0 - 1) >> 1;
    const bool fy = j <= 2 || j >= g.Ny - 1, fz = k <= 2 || k >= g.Nz - 1;
    const long long nd = ((long long)(k - 1) * g.Ny + (j - 1)) * L.P + c0;
    // i = lo .. hi of the row are active
    auto block = [&](int q, bool row, int lo, int hi) {
        if (!row || c0 + W - 1 < lo || c0 > hi) return;
        const MGBlockDesc& cb = C.blk[q - S::Q0];
        const T* cr = xc + cb.off + (long long)J * cb.n1 + (long long)K * cb.n1 * cb.n2;
        Packet* xp = reinterpret_cast<Packet*>(x + q * L.comp + nd);
        Packet v = *xp;
        T c[W / 2 + 1];
#pragma unroll
        for (int e = 0; e <= W / 2; e++) c[e] = I0 + e >= 0 && I0 + e < cb.n1 ? cr[I0 + e] : T(0);
#pragma unroll
        for (int e = 0; e < W; e++)
            if (c0 + e >= lo && c0 + e <= hi) v.v[e] += alpha * c[(e + 1) / 2];
        *xp = v;
    };
    if (S::A) {
        block(0, !fy && !fz, 2, g.xs - 1);
        block(1, !fz && j > 1 && j < g.ys, 3, g.Nx - 2);
        block(2, !fy && k > 1 && k < g.zs, 3, g.Nx - 2);
    }
    if (S::V) block(3, !fy && !fz, 3, g.Nx - 2);
}

template <typename T, int KIND, int QS = 0>
static size_t mg0_smem() {
    return PLTiles<T, MG0Set<QS>::NQ, MG0Set<QS>::NC, typename MG0Coef<T>::type>::SMEM;
}

// raise the dynamic shared-memory limit of the level-0 kernels once per device
template <typename T>
static void mg0_prepare() {
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    auto one = [](auto uni, auto rows) {
        constexpr bool U = decltype(uni)::value;
        constexpr int R = decltype(rows)::value;
#define ATTR(K, Q) \
    cudaFuncSetAttribute(mg0_tiled<T, K, Q, U, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mg0_smem<T, K, Q>())
    ATTR(0, 0); ATTR(1, 0); ATTR(2, 0);
    ATTR(0, 1); ATTR(1, 1); ATTR(2, 1);
    ATTR(0, 2); ATTR(1, 2); ATTR(2, 2);
        if constexpr (sizeof(T) == 4) { ATTR(3, 1); ATTR(3, 2); }
#undef ATTR
    };
    using R1 = std::integral_constant<int, 1>;
    one(std::true_type(), R1());
    one(std::false_type(), R1());
    if constexpr (sizeof(T) == 4) {
        using R2 = std::integral_constant<int, 2>;
        one(std::true_type(), R2());
        one(std::false_type(), R2());
    }
    cudaFuncSetAttribute(mg_sub<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, MGC_SMEM);
    cudaFuncSetAttribute(mg_sub<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    done.fetch_or(bit, std::memory_order_acq_rel);
}

// log2 of the CTAs of the coarse sub-cycle's clusters: 16 where the device can place such a cluster with the most
// shared memory it may take, else 8
template <typename T>
static int mgc_size() {
    mg0_prepare<T>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(MGC_THREADS);
    cfg.dynamicSmemBytes = MGC_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {16, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, mg_sub<T>, &cfg) == cudaSuccess && n >= 1) return 4;
    cudaGetLastError();
    return 3;
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// Cyclic Jacobi eigen-decomposition of a symmetric m x m matrix (row-major, in
// place): on return A's diagonal holds the eigenvalues and V the eigenvectors
// (columns).
static void sym_eig_jacobi(int m, std::vector<double>& A, std::vector<double>& V) {
    V.assign((size_t)m * m, 0.0);
    for (int q = 0; q < m; q++) V[(size_t)q * m + q] = 1.0;
    for (int sweep = 0; sweep < 60; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int p = 0; p < m; p++)
            for (int q = 0; q < m; q++) {
                double a = A[(size_t)p * m + q];
                tot += a * a;
                if (p != q) off += a * a;
            }
        if (off <= 1e-30 * tot) break;
        for (int p = 0; p < m - 1; p++)
            for (int q = p + 1; q < m; q++) {
                const double apq = A[(size_t)p * m + q];
                if (std::fabs(apq) < 1e-300) continue;
                const double app = A[(size_t)p * m + p], aqq = A[(size_t)q * m + q];
                const double th = (aqq - app) / (2.0 * apq);
                const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
                const double c = 1.0 / std::sqrt(t * t + 1.0), sn = t * c;
                for (int k = 0; k < m; k++) {       // columns p, q
                    double akp = A[(size_t)k * m + p], akq = A[(size_t)k * m + q];
                    A[(size_t)k * m + p] = c * akp - sn * akq;
                    A[(size_t)k * m + q] = sn * akp + c * akq;
                }
                for (int k = 0; k < m; k++) {       // rows p, q
                    double apk = A[(size_t)p * m + k], aqk = A[(size_t)q * m + k];
                    A[(size_t)p * m + k] = c * apk - sn * aqk;
                    A[(size_t)q * m + k] = sn * apk + c * aqk;
                }
                for (int k = 0; k < m; k++) {
                    double vkp = V[(size_t)k * m + p], vkq = V[(size_t)k * m + q];
                    V[(size_t)k * m + p] = c * vkp - sn * vkq;
                    V[(size_t)k * m + q] = sn * vkp + c * vkq;
                }
            }
    }
}
#define CKM(call)                                                                        \
    do {                                                                                 \
        cudaError_t _e = (call);                                                         \
        if (_e != cudaSuccess) {                                                         \
            err = std::string(#call) + ": " + cudaGetErrorString(_e);                    \
            return -2;                                                                   \
        }                                                                                \
    } while (0)

static inline unsigned nblk(long long n) { return (unsigned)((n + 255) / 256); }

template <typename T>
QmsMG<T>::~QmsMG() { release(); }

template <typename T>
void QmsMG<T>::release() {
    for (auto& L : lv) {
        T* ps[] = {L.w1, L.w2, L.w3, L.dg, L.dinv, L.x, L.b, L.t, L.mass};
        for (T* p : ps) if (p) cudaFree(p);
    }
    lv.clear();
    views[1].clear();
    views[2].clear();
    if (dminv) cudaFree(dminv);
    if (dmoff) cudaFree(dmoff);
    dminv = nullptr; dmoff = nullptr;
}

template <typename T>
int QmsMG<T>::levels_for(const QGrid& g, int min_coarse) {
    int dims[4][3] = {{g.xs, g.Ny, g.Nz}, {g.Nx, g.ys, g.Nz}, {g.Nx, g.Ny, g.zs}, {g.Nx, g.Ny, g.Nz}};
    int n = 0;
    for (;;) {
        n++;
        int mx = 0;
        for (int b = 0; b < 4; b++) mx = std::max({mx, dims[b][0], dims[b][1], dims[b][2]});
        if (mx <= min_coarse || n >= 12) return n;
        for (int b = 0; b < 4; b++) for (int a = 0; a < 3; a++) dims[b][a] = (dims[b][a] + 1) / 2;
    }
}

template <typename T>
size_t QmsMG<T>::bytes_for(const QGrid& g, int min_coarse, bool tiled) {
    // every level stores 9 values per point; a tiled level 0 (stored node coefficients,
    // more than one level) stores none: its x/b are the Krylov vectors and the caller's temporary
    long long dims[4][3] = {{g.xs, g.Ny, g.Nz}, {g.Nx, g.ys, g.Nz}, {g.Nx, g.Ny, g.zs}, {g.Nx, g.Ny, g.Nz}};
    size_t total = 0;
    for (int l = 0; l < 16; l++) {
        long long pts = 0, mx = 0;
        for (int b = 0; b < 4; b++) {
            pts += dims[b][0] * dims[b][1] * dims[b][2];
            mx = std::max({mx, dims[b][0], dims[b][1], dims[b][2]});
        }
        if (mx <= min_coarse) {
            total += (size_t)pts * 9 * sizeof(T);
            total += (size_t)4 * pts * pts * 8 / 4 + 1024;
            break;
        }
        if (!(tiled && l == 0)) total += (size_t)pts * 9 * sizeof(T);
        for (int b = 0; b < 4; b++) for (int a = 0; a < 3; a++) dims[b][a] = (dims[b][a] + 1) / 2;
    }
    return total;
}

template <typename T>
int QmsMG<T>::build(const QGrid& g, const QCoef<T>& c, const QStepPar<T>& P, T vshift, cudaStream_t st) {
    release();
    // level sizes
    int dims[4][3] = {{g.xs, g.Ny, g.Nz}, {g.Nx, g.ys, g.Nz}, {g.Nx, g.Ny, g.zs}, {g.Nx, g.Ny, g.Nz}};
    for (;;) {
        MGLevelDev<T> L{};
        L.nb = 4;
        long long off = 0;
        int mx = 0;
        for (int b = 0; b < 4; b++) {
            L.blk[b].n1 = dims[b][0]; L.blk[b].n2 = dims[b][1]; L.blk[b].n3 = dims[b][2];
            L.blk[b].off = off;
            off += (long long)dims[b][0] * dims[b][1] * dims[b][2];
            mx = std::max({mx, dims[b][0], dims[b][1], dims[b][2]});
        }
        L.total = off;
        lv.push_back(L);
        if (mx <= min_coarse || (int)lv.size() >= max_levels) break;
        for (int b = 0; b < 4; b++) for (int a = 0; a < 3; a++) dims[b][a] = (dims[b][a] + 1) / 2;
    }
    // With stored node coefficients level 0 runs on node tiles (mg0_tiled) and level 1 is
    // coarsened straight from the coefficients: level 0 keeps no arrays.
    tiled0 = lv.size() > 1 && c.nc != nullptr;
    if (!tiled0) {
        err = "multigrid needs at least two levels and stored node coefficients";
        release();
        return -1;
    }
    for (size_t l = tiled0 ? 1 : 0; l < lv.size(); l++) {
        MGLevelDev<T>& L = lv[l];
        const size_t bytes = L.total * sizeof(T);
        CKM(cudaMalloc(&L.w1, bytes)); CKM(cudaMalloc(&L.w2, bytes)); CKM(cudaMalloc(&L.w3, bytes));
        CKM(cudaMalloc(&L.dg, bytes)); CKM(cudaMalloc(&L.dinv, bytes)); CKM(cudaMalloc(&L.t, bytes));
        CKM(cudaMalloc(&L.mass, bytes));
        if (l > 0) { CKM(cudaMalloc(&L.x, bytes)); CKM(cudaMalloc(&L.b, bytes)); }
        // the restriction leaves out aggregates of Dirichlet points alone: their right-hand side is zero
        if (l == 1) CKM(cudaMemsetAsync(L.b, 0, bytes, st));
    }
    g0 = g; c0 = c; P0 = P; vshift0 = vshift;
    g0grid = qms_pl_tiles(g);
    const double ncut = vcut > 0.0 ? vcut : (sizeof(T) == 8 ? 1e-9 : 1e-5);
    mg_coarsen_fine<<<nblk(lv[1].total), 256, 0, st>>>(g, c, P, vshift, lv[0], lv[1], ncut);
    mg_mask_links<<<nblk(lv[1].total), 256, 0, st>>>(lv[1]);
    for (size_t l = tiled0 ? 2 : 1; l < lv.size(); l++) {
        mg_coarsen<<<nblk(lv[l].total), 256, 0, st>>>(lv[l - 1], lv[l], ncut);
        mg_mask_links<<<nblk(lv[l].total), 256, 0, st>>>(lv[l]);
    }
    CKM(cudaGetLastError());
    // coarsest level: dense inverse per block in FP64 on the host
    MGLevelDev<T>& C = lv.back();
    std::vector<T> w1(C.total), w2(C.total), w3(C.total), dg(C.total), dinv(C.total), mass(C.total);
    CKM(cudaMemcpyAsync(mass.data(), C.mass, C.total * sizeof(T), cudaMemcpyDeviceToHost, st));
    CKM(cudaMemcpyAsync(w1.data(), C.w1, C.total * sizeof(T), cudaMemcpyDeviceToHost, st));
    CKM(cudaMemcpyAsync(w2.data(), C.w2, C.total * sizeof(T), cudaMemcpyDeviceToHost, st));
    CKM(cudaMemcpyAsync(w3.data(), C.w3, C.total * sizeof(T), cudaMemcpyDeviceToHost, st));
    CKM(cudaMemcpyAsync(dg.data(), C.dg, C.total * sizeof(T), cudaMemcpyDeviceToHost, st));
    CKM(cudaMemcpyAsync(dinv.data(), C.dinv, C.total * sizeof(T), cudaMemcpyDeviceToHost, st));
    CKM(cudaStreamSynchronize(st));
    std::vector<long long> moff(C.nb);
    long long mtot = 0;
    for (int b = 0; b < C.nb; b++) {
        long long m = (long long)C.blk[b].n1 * C.blk[b].n2 * C.blk[b].n3;
        moff[b] = mtot;
        mtot += m * m;
    }
    std::vector<double> minv(mtot, 0.0);
    for (int b = 0; b < C.nb; b++) {
        const MGBlockDesc& B = C.blk[b];
        const int m = B.n1 * B.n2 * B.n3;
        std::vector<double> A((size_t)m * m, 0.0), Inv((size_t)m * m, 0.0);
        for (int r = 0; r < m; r++) {
            long long t = B.off + r;
            Inv[(size_t)r * m + r] = 1.0;
            if (dinv[t] == T(0)) { A[(size_t)r * m + r] = 1.0; continue; }
            A[(size_t)r * m + r] = dg[t];
            int i = r % B.n1, j = (r / B.n1) % B.n2, k = r / (B.n1 * B.n2);
            auto link = [&](int nb, T w) { if (w != T(0)) A[(size_t)r * m + nb] -= w; };
            if (i > 0) link(r - 1, w1[t - 1]);
            if (i + 1 < B.n1) link(r + 1, w1[t]);
            if (j > 0) link(r - B.n1, w2[t - B.n1]);
            if (j + 1 < B.n2) link(r + B.n1, w2[t]);
            if (k > 0) link(r - B.n1 * B.n2, w3[t - (long long)B.n1 * B.n2]);
            if (k + 1 < B.n3) link(r + B.n1 * B.n2, w3[t]);
        }
        if (b == C.nb - 1) {
            // V block: pseudo-inverse.  An isolated conductor's potential is pinned only by the
            // 1e-12 S/m floor; on the coarsest grid that is an eigenvalue ~1e-19 of the operator
            // scaled by the summed level-0 diagonals of each point (its stiffness).  Inverting it
            // would amplify round-off without bound, so eigenvalues at or below the cut are
            // dropped (the mode does not enter A or H), and so are the near-null points the
            // coarsening already took out (inactive rows).  Scaling by the point's own Galerkin
            // diagonal instead would hide the mode: a body that collapsed into one point has a
            // diagonal of pure rounding noise and an eigenvalue near 1 in that scaling.
            std::vector<double> dsq(m);
            for (int r = 0; r < m; r++) {
                const long long t = B.off + r;
                dsq[r] = dinv[t] == T(0) ? 1.0 : 1.0 / std::sqrt(std::fabs((double)mass[t]));
            }
            for (int r = 0; r < m; r++)
                for (int q = 0; q < m; q++) A[(size_t)r * m + q] *= dsq[r] * dsq[q];
            for (int r = 0; r < m; r++)             // symmetrise round-off
                for (int q = r + 1; q < m; q++) {
                    double av = 0.5 * (A[(size_t)r * m + q] + A[(size_t)q * m + r]);
                    A[(size_t)r * m + q] = A[(size_t)q * m + r] = av;
                }
            std::vector<double> Q;
            sym_eig_jacobi(m, A, Q);
            for (int r = 0; r < m; r++)
                for (int q = 0; q < m; q++) {
                    double acc = 0.0;
                    for (int e = 0; e < m; e++) {
                        const double lam = A[(size_t)e * m + e];
                        if (lam > ncut) acc += Q[(size_t)r * m + e] * Q[(size_t)q * m + e] / lam;
                    }
                    const bool off_r = dinv[B.off + r] == T(0), off_q = dinv[B.off + q] == T(0);
                    Inv[(size_t)r * m + q] = off_r || off_q ? 0.0 : dsq[r] * acc * dsq[q];
                }
            std::memcpy(&minv[moff[b]], Inv.data(), sizeof(double) * (size_t)m * m);
            continue;
        }
        // A blocks: Gauss-Jordan with partial pivoting
        for (int col = 0; col < m; col++) {
            int piv = col;
            for (int r = col + 1; r < m; r++)
                if (std::fabs(A[(size_t)r * m + col]) > std::fabs(A[(size_t)piv * m + col])) piv = r;
            if (A[(size_t)piv * m + col] == 0.0) { err = "singular coarsest-level operator"; return -1; }
            if (piv != col)
                for (int q = 0; q < m; q++) {
                    std::swap(A[(size_t)piv * m + q], A[(size_t)col * m + q]);
                    std::swap(Inv[(size_t)piv * m + q], Inv[(size_t)col * m + q]);
                }
            const double p = 1.0 / A[(size_t)col * m + col];
            for (int q = 0; q < m; q++) { A[(size_t)col * m + q] *= p; Inv[(size_t)col * m + q] *= p; }
            for (int r = 0; r < m; r++) {
                if (r == col) continue;
                const double f = A[(size_t)r * m + col];
                if (f == 0.0) continue;
                for (int q = 0; q < m; q++) {
                    A[(size_t)r * m + q] -= f * A[(size_t)col * m + q];
                    Inv[(size_t)r * m + q] -= f * Inv[(size_t)col * m + q];
                }
            }
        }
        std::memcpy(&minv[moff[b]], Inv.data(), sizeof(double) * (size_t)m * m);
    }
    CKM(cudaMalloc(&dminv, std::max<long long>(mtot, 1) * 8));
    CKM(cudaMalloc(&dmoff, C.nb * sizeof(long long)));
    CKM(cudaMemcpyAsync(dminv, minv.data(), mtot * 8, cudaMemcpyHostToDevice, st));
    CKM(cudaMemcpyAsync(dmoff, moff.data(), C.nb * sizeof(long long), cudaMemcpyHostToDevice, st));
    CKM(cudaStreamSynchronize(st));
    // views of the three A blocks and of the V block, for cycles on one side of the A-V
    // coupling: same arrays, block table and pointers restricted to those blocks
    views[1].assign(lv.begin(), lv.end());
    views[2].assign(lv.begin(), lv.end());
    for (size_t l = 0; l < lv.size(); l++) {
        const long long o = lv[l].blk[3].off;
        MGLevelDev<T>& A = views[1][l];
        A.nb = 3;
        A.total = o;
        MGLevelDev<T>& V = views[2][l];
        V.nb = 1;
        V.blk[0] = lv[l].blk[3];
        V.blk[0].off = 0;
        V.total = lv[l].total - o;
        T** ps[] = {&V.w1, &V.w2, &V.w3, &V.dg, &V.dinv, &V.x, &V.b, &V.t, &V.mass};
        for (T** q : ps)
            if (*q) *q += o;
    }
    // the first level of each view's sub-cycle in one launch: as many levels as fit shared memory (and
    // tail_points allows)
    sub_lg = mgc_size<T>();
    for (int qs = 0; qs < 3; qs++) {
        const std::vector<MGLevelDev<T>>& v = qs == 0 ? lv : views[qs];
        auto smem = [&](int lt) {
            size_t most = 0;
            for (int b = 0; b < v[lt].nb; b++) {
                const MGBlockDesc& c = v.back().blk[b];
                size_t bytes = (size_t)c.n1 * c.n2 * c.n3 * sizeof(double);
                for (size_t l = lt; l < v.size(); l++)
                    bytes += (size_t)mgc_len(v[l].blk[b], sub_lg, l + 1 < v.size()) * sizeof(T);
                most = std::max(most, bytes);
            }
            return most;
        };
        auto fits = [&](int lt) {
            for (int b = 0; b < v[lt].nb; b++) {
                const MGBlockDesc& B = v[lt].blk[b];
                const long long pts = (long long)B.n1 * B.n2 * B.n3;
                if (tail_points < 0 || (tail_points > 0 && pts > tail_points)) return false;
            }
            return smem(lt) <= MGC_SMEM;
        };
        int lt = (int)v.size() - 1;              // (the coarsest level, 5^3 points a block at most, always fits)
        while (lt > 1 && (int)v.size() - (lt - 1) <= MGC_LEVELS && fits(lt - 1)) lt--;
        sub_first[qs] = lt;
        sub_smem[qs] = smem(lt);
    }
    return 0;
}

// z = MG(r): level-0 right-hand side b0 (scaled pointwise by `bscale` when given),
// result in x0; t0 is a level-0 temporary.  Returns the number of kernel launches.
template <typename T>
int QmsMG<T>::vcycle(const T* b0, bool scaled, T* x0, const CUtensorMap& x0map, T* t0, const CUtensorMap& t0map,
                     const CUtensorMap& cmap, unsigned* err, cudaStream_t st, int qs,
                     const CUtensorMap* b0map) {
    if (qs == 1) return vcycle_q<1>(b0, scaled, x0, x0map, t0, t0map, cmap, err, st, b0map);
    if (qs == 2) return vcycle_q<2>(b0, scaled, x0, x0map, t0, t0map, cmap, err, st, b0map);
    return vcycle_q<0>(b0, scaled, x0, x0map, t0, t0map, cmap, err, st, nullptr);
}

template <typename T>
template <int QS>
int QmsMG<T>::vcycle_q(const T* b0, bool scaled, T* x0, const CUtensorMap& x0map, T* t0, const CUtensorMap& t0map,
                       const CUtensorMap& cmap, unsigned* err, cudaStream_t st,
                       const CUtensorMap* b0map) {
    int launches = 0;
    std::vector<MGLevelDev<T>>& lv = QS == 0 ? this->lv : views[QS];   // levels >= 1 of the cycle's blocks
    const long long* dmo = dmoff + (QS == 2 ? 3 : 0);                    // their dense coarsest inverses
    const int nl = (int)lv.size();
    // sweeps on each side: the V-block cycle may use its own count
    const int n1 = (QS == 2 && nu_v > 0) ? nu_v : nu1, n2 = (QS == 2 && nu_v > 0) ? nu_v : nu2;
    const int sc = scaled ? 1 : 0;
    mg0_prepare<T>();
    struct Buf { T* p; const CUtensorMap* m; };
    // level-0 sweeps: KIND 0 writes XO from b; KIND 1 reads XI (tile copies) and writes XO;
    // KIND 2 reads XI and writes the level-1 right-hand side
#define MG0U(KIND, XI, XO, BC, OM, OM1, UNI, ROWS)                                                               \
    pdl_launch(mg0_tiled<T, KIND, QS, UNI, ROWS>, g0grid, dim3(OTX, OTY / ROWS), mg0_smem<T, KIND, QS>(), st, 0,  \
               g0, P0, vshift0, (OM), (OM1), b0, sc, *(XI).m, cmap, (XO), lv[1], (BC), err)
#define MG0(KIND, XI, XO, BC, OM, OM1)                                                                           \
    do {                                                                                                          \
        if (ROWS2 > 1 && two) {                                                                                   \
            if (cubic) MG0U(KIND, XI, XO, BC, OM, OM1, true, ROWS2);                                             \
            else MG0U(KIND, XI, XO, BC, OM, OM1, false, ROWS2);                                                  \
        } else {                                                                                                  \
            if (cubic) MG0U(KIND, XI, XO, BC, OM, OM1, true, 1);                                                 \
            else MG0U(KIND, XI, XO, BC, OM, OM1, false, 1);                                                      \
        }                                                                                                         \
    } while (0)
    // rows per thread: two on grids of many tiles (FP32)
    constexpr int ROWS2 = sizeof(T) == 4 ? 2 : 1;
    constexpr bool FIRST2 = sizeof(T) == 4;      // (FP64 callers hand over no map of b)
    const bool two = (long long)g0grid.x * g0grid.y * g0grid.z >= QMS_CTA_TARGET;
    auto wgt = [&](int s, int nu) { return mg_weight<T>(omega, s, nu); };
    const bool cubic = P0.idx2 == P0.idy2 && P0.idx2 == P0.idz2;
    // level 0: nu1 + nu2 sweeps alternate between x0 and t0 (the prolongation is in place);
    // start in t0 when that count is even so that the last write lands in x0
    Buf x{x0, &x0map}, t{t0, &t0map};
    if ((n1 + n2) % 2 == 0) std::swap(x, t);
    int s = 1;
    if constexpr (FIRST2 && QS != 0) {
        if (b0map && scaled && n1 >= 2) {
            // the first two sweeps in one pass, from b's tiles (KIND 3), into the buffer the second
            // sweep writes
            Buf bb{const_cast<T*>(b0), b0map};
            MG0(3, bb, t.p, nullptr, wgt(1, n1), wgt(0, n1));
            std::swap(x, t);
            launches++;
            s = 2;
        }
    }
    if (s == 1) {
        MG0(0, x, x.p, nullptr, wgt(0, n1), T(0));
        launches++;
    }
    // the A-block sweeps are the largest single kernel of a transient step: optionally timed,
    // with their algorithmic bytes (x and b read, x written, one material byte per cell)
    const double asweep_bytes = 3.0 * sizeof(T) * (double)g0.oV + (double)g0.xs * g0.ys * g0.zs;
    auto sweep = [&](Buf& xi, T* xo, T om) {
        void* tok = (QS == 1 && prof) ? prof->begin(MGPROF_A_SWEEP, asweep_bytes) : nullptr;
        MG0(1, xi, xo, nullptr, om, T(0));
        if (tok) prof->end(tok);
    };
    for (; s < n1; s++) {
        sweep(x, t.p, wgt(s, n1));
        std::swap(x, t);
        launches++;
    }
    MG0(2, x, nullptr, lv[1].b, omega, T(0));
    launches++;
    // levels >= 1: nu_coarse sweeps on each side when set
    const int nuc1 = (QS == 2 && nu_v > 0) ? nu_v : (nu_coarse > 0 ? nu_coarse : nu1);
    const int nuc2 = (QS == 2 && nu_v > 0) ? nu_v : (nu_coarse > 0 ? nu_coarse : nu2);
    // from level lt on the whole sub-cycle is one launch
    const int lt = sub_first[QS];
    for (int l = 1; l < nl; l++) {
        MGLevelDev<T>& L = lv[l];
        if (l == lt) {
            MGSub<T> sub{};
            sub.nl = nl - lt;
            sub.lg = sub_lg;
            for (int q = 0; q < MGC_SWEEPS; q++) { sub.w1[q] = wgt(q, nuc1); sub.w2[q] = wgt(q, nuc2); }
            for (int q = 0; q < sub.nl; q++) sub.L[q] = lv[lt + q];
            pdl_launch(mg_sub<T>, dim3(L.nb << sub_lg), dim3(MGC_THREADS), sub_smem[QS], st, 1u << sub_lg, sub, dminv, dmo,
                       alpha, nuc1, nuc2);
            launches++;
            break;
        }
        T* xl = L.x;
        T* tl = L.t;
        if (nuc1 >= 2) {
            pdl_launch(mg_smooth01<T>, dim3(nblk(L.total)), dim3(256), 0, st, 0, L, L.b, wgt(0, nuc1), wgt(1, nuc1), xl);
        } else {
            pdl_launch(mg_smooth0<T>, dim3(nblk(L.total)), dim3(256), 0, st, 0, L, L.b, wgt(0, nuc1), xl);
        }
        launches++;
        for (int s = 2; s < nuc1; s++) {
            pdl_launch(mg_smooth<T>, dim3(nblk(L.total)), dim3(256), 0, st, 0, L, L.b, wgt(s, nuc1), xl, tl);
            std::swap(xl, tl);
            launches++;
        }
        L.x = xl;
        L.t = tl;
        int e1 = 0, e2 = 0, e3 = 0;
        for (int q = 0; q < L.nb; q++) {
            e1 = std::max(e1, L.blk[q].n1);
            e2 = std::max(e2, L.blk[q].n2);
            e3 = std::max(e3, L.blk[q].n3);
        }
        const int xt = (e1 + MGR_X - 1) / MGR_X;
        pdl_launch(mg_restrict<T>, dim3(L.nb * xt, (e2 + MGR_Y - 1) / MGR_Y, (e3 + MGR_Z - 1) / MGR_Z),
                   dim3(MGR_X, MGR_Y, MGR_Z), 0, st, 0, L, L.b, xl, lv[l + 1], lv[l + 1].b, xt);
        launches++;
    }
    for (int l = lt - 1; l >= 1; l--) {
        MGLevelDev<T>& L = lv[l];
        T* xl = L.x;
        T* tl = L.t;
        pdl_launch(mg_prolong_smooth<T>, dim3(nblk(L.total)), dim3(256), 0, st, 0, L, L.b, wgt(0, nuc2), xl, tl, lv[l + 1],
                   lv[l + 1].x, alpha);
        std::swap(xl, tl);
        launches++;
        for (int s = 1; s < nuc2; s++) {
            pdl_launch(mg_smooth<T>, dim3(nblk(L.total)), dim3(256), 0, st, 0, L, L.b, wgt(s, nuc2), xl, tl);
            std::swap(xl, tl);
            launches++;
        }
        L.x = xl;
        L.t = tl;
    }
    const int cols = MGP_X * 16 / (int)sizeof(T);
    pdl_launch(mg0_prolong<T, QS>, dim3((g0.xs + cols - 1) / cols, (g0.ys + MGP_Y - 1) / MGP_Y, g0.Nz),
               dim3(MGP_X, MGP_Y), 0, st, 0, g0, x.p, lv[1], lv[1].x, alpha);
    launches++;
    for (int s = 0; s < n2; s++) {
        sweep(x, t.p, wgt(s, n2));
        std::swap(x, t);
        launches++;
    }
#undef MG0
#undef MG0U
    return launches;
}

template struct QmsMG<float>;
template struct QmsMG<double>;

// ---------------------------------------------------------------------------
// conductor-region coarse space of the V block
// ---------------------------------------------------------------------------
namespace {

// y = K^+ s with s[r] the sum over the V rows of region r of b * bscale, FP64 in a fixed order: a CTA
// per chunk of at most QMS_REGION_CHUNK rows of one region (a CTA per region left the largest body to
// one SM: 12 us at 48^3, 27 us at 128^3; runs of steps 96^3 213 -> 202 ms, 128^3 254 -> 244), the chunks of each region and the K x K product in the CTA
// that arrives last.
#define QMS_REGION_CHUNK 1024
template <typename T>
__global__ void __launch_bounds__(256) qk_region_solve(const int* __restrict__ cptr, const int* __restrict__ rchunk,
                                                      const int* __restrict__ rows, const T* b,
                                                      const float* __restrict__ bscale, double* part, int K,
                                                      const double* __restrict__ Kp, double* y,
                                                      unsigned* counter) {
    __shared__ double sh[32], s[QMS_REGION_MAX];
    __shared__ bool lastcta;
    double acc = 0.0;
    pdl_wait();
    for (int e = cptr[blockIdx.x] + threadIdx.x; e < cptr[blockIdx.x + 1]; e += blockDim.x) {
        const int row = rows[e];
        acc += (double)b[row] * (bscale ? (double)bscale[row] : 1.0);
    }
    acc = qBlockSum(acc, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = acc;
        __threadfence();
        lastcta = atomicAdd(counter, 1u) == gridDim.x - 1;
        if (lastcta) *counter = 0;
    }
    __syncthreads();
    if (!lastcta) return;
    __threadfence();
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < K; r += blockDim.x >> 5) {
        double t = 0.0;
        for (int q = rchunk[r] + lane; q < rchunk[r + 1]; q += 32) t += __ldcg(part + q);
        t = qWarpSum(t);
        if (lane == 0) s[r] = t;
    }
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < K; r += blockDim.x >> 5) {
        double t = 0.0;
        for (int q = lane; q < K; q += 32) t += Kp[(long long)r * K + q] * s[q];
        t = qWarpSum(t);
        if (lane == 0) y[r] = t;
    }
}

// z[row] += y[region of row]
template <typename T>
__global__ void qk_region_scatter(int total, const int* __restrict__ rows, const int* __restrict__ rid,
                                  const double* y, T* z) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (e < total) z[rows[e]] += (T)y[rid[e]];
}

}  // namespace

QmsRegions::~QmsRegions() { release(); }

void QmsRegions::release() {
    void* ps[] = {cptr, rchunk, rows, rid, Kp, part, y, counter};
    for (void* p : ps) if (p) cudaFree(p);
    cptr = rchunk = rows = rid = nullptr;
    Kp = part = y = nullptr;
    counter = nullptr;
    K = nchunk = 0;
}

int QmsRegions::build(const QGrid& g, const uint8_t* slots, const double* rows6, int nmat, double vshift,
                      double cut, cudaStream_t st) {
    release();
    const int xs = g.xs, ys = g.ys, zs = g.zs, Nx = g.Nx, Ny = g.Ny, Nz = g.Nz;
    const long long ncell = (long long)xs * ys * zs;
    // per-slot conductivity per axis and its maximum (slot 0: vacuum)
    std::vector<double> sax(3 * (nmat + 1), 0.0), smax(nmat + 1, 0.0);
    for (int r = 0; r < nmat; r++)
        for (int a = 0; a < 3; a++) {
            sax[3 * (r + 1) + a] = rows6[r * 6 + 3 + a];
            smax[r + 1] = std::max(smax[r + 1], rows6[r * 6 + 3 + a]);
        }
    auto cid = [&](int i, int j, int k) { return (long long)(i - 1) + (long long)(j - 1) * xs + (long long)(k - 1) * xs * ys; };
    auto is_cond = [&](long long c) { return smax[slots[c]] > 1.0; };
    // connected bodies: union-find over conductor cells of one slot (6-neighbours)
    std::vector<int> par(ncell, -1);                 // ncell < 2^31 (checked at creation)
    auto find = [&](long long a) -> long long {
        while (par[a] != a) { par[a] = par[par[a]]; a = par[a]; }
        return a;
    };
    for (int k = 1; k <= zs; k++)
        for (int j = 1; j <= ys; j++)
            for (int i = 1; i <= xs; i++) {
                const long long c = cid(i, j, k);
                if (!is_cond(c)) continue;
                par[c] = (int)c;
                const long long nb[3] = {i > 1 ? cid(i - 1, j, k) : -1, j > 1 ? cid(i, j - 1, k) : -1,
                                         k > 1 ? cid(i, j, k - 1) : -1};
                for (long long q : nb)
                    if (q >= 0 && par[q] >= 0 && slots[q] == slots[c]) {
                        const long long ra = find(c), rb = find(q);
                        if (ra != rb) par[std::max(ra, rb)] = (int)std::min(ra, rb);
                    }
            }
    // region of each active V node: body of its incident conductor cell with the largest sigma
    const long long Nn = g.Nn;
    std::vector<int> nreg(Nn, -1);
    std::vector<long long> roots;                   // region index -> body root
    std::vector<long long> count;
    std::map<long long, int> rmap;
    for (int k = 1; k <= Nz; k++)
        for (int j = 1; j <= Ny; j++)
            for (int i = 1; i <= Nx; i++) {
                if (qFixV(g, i, j, k)) continue;
                double best = -1.0;
                long long broot = -1;
                for (int ck = k - 1; ck <= k; ck++)
                    for (int cj = j - 1; cj <= j; cj++)
                        for (int ci = i - 1; ci <= i; ci++) {
                            if (ci < 1 || cj < 1 || ck < 1 || ci > xs || cj > ys || ck > zs) continue;
                            const long long c = cid(ci, cj, ck);
                            if (!is_cond(c)) continue;
                            const long long rt = find(c);
                            const double sv = smax[slots[c]];
                            if (sv > best || (sv == best && rt < broot)) { best = sv; broot = rt; }
                        }
                if (broot < 0) continue;
                auto it = rmap.find(broot);
                int r;
                if (it == rmap.end()) {
                    r = (int)roots.size();
                    rmap[broot] = r;
                    roots.push_back(broot);
                    count.push_back(0);
                } else {
                    r = it->second;
                }
                count[r]++;
                nreg[(i - 1) + (long long)(j - 1) * Nx + (long long)(k - 1) * Nx * Ny] = r;
            }
    int nr = (int)roots.size();
    if (nr == 0) return 0;
    // keep at most QMS_REGION_MAX regions (the largest; ties by first appearance)
    std::vector<int> order(nr), newid(nr, -1);
    for (int r = 0; r < nr; r++) order[r] = r;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return count[a] > count[b]; });
    const int Kr = std::min(nr, QMS_REGION_MAX);
    std::vector<int> keep(order.begin(), order.begin() + Kr);
    std::sort(keep.begin(), keep.end());
    for (int q = 0; q < Kr; q++) newid[keep[q]] = q;
    for (long long p = 0; p < Nn; p++)
        if (nreg[p] >= 0) nreg[p] = newid[nreg[p]];
    // Galerkin matrix W^T A_V W from the links crossing region boundaries (no cancellation):
    // link weight max(sigma_edge, floor) / h^2, sigma_edge the mean of the four cells around it
    const double floor_s = (double)1.0e-12f;
    const double ih2[3] = {1.0 / (g.dx * g.dx), 1.0 / (g.dy * g.dy), 1.0 / (g.dz * g.dz)};
    std::vector<double> Km((size_t)Kr * Kr, 0.0);
    std::vector<double> Tr(Kr, 0.0);              // sum of the V-operator diagonal over each region
    auto sig_edge = [&](int a, int i, int j, int k) {
        // edge from node (i,j,k) along axis a: cells with that axis index i/j/k and the other two
        // indices in {n-1, n}
        double acc = 0.0;
        for (int u = 0; u < 2; u++)
            for (int v = 0; v < 2; v++) {
                int ci = i, cj = j, ck = k;
                if (a == 0) { cj = j - 1 + u; ck = k - 1 + v; }
                else if (a == 1) { ci = i - 1 + u; ck = k - 1 + v; }
                else { ci = i - 1 + u; cj = j - 1 + v; }
                if (ci < 1 || cj < 1 || ck < 1 || ci > xs || cj > ys || ck > zs) continue;
                acc += sax[3 * slots[cid(ci, cj, ck)] + a];
            }
        return 0.25 * acc;
    };
    for (int k = 1; k <= Nz; k++)
        for (int j = 1; j <= Ny; j++)
            for (int i = 1; i <= Nx; i++) {
                const long long p = (i - 1) + (long long)(j - 1) * Nx + (long long)(k - 1) * Nx * Ny;
                for (int a = 0; a < 3; a++) {
                    const int i2 = i + (a == 0), j2 = j + (a == 1), k2 = k + (a == 2);
                    if (i2 > Nx || j2 > Ny || k2 > Nz) continue;
                    const long long q = (i2 - 1) + (long long)(j2 - 1) * Nx + (long long)(k2 - 1) * Nx * Ny;
                    const int R = nreg[p], S = nreg[q];
                    if (R < 0 && S < 0) continue;
                    const double w = std::max(sig_edge(a, i, j, k), floor_s) * ih2[a];
                    if (R >= 0) Tr[R] += (1.0 + vshift) * w;
                    if (S >= 0) Tr[S] += (1.0 + vshift) * w;
                    if (vshift != 0.0) {
                        if (R >= 0) Km[(size_t)R * Kr + R] += vshift * w;
                        if (S >= 0) Km[(size_t)S * Kr + S] += vshift * w;
                    }
                    if (R == S) continue;
                    if (R >= 0) Km[(size_t)R * Kr + R] += w;
                    if (S >= 0) Km[(size_t)S * Kr + S] += w;
                    if (R >= 0 && S >= 0) {
                        Km[(size_t)R * Kr + S] -= w;
                        Km[(size_t)S * Kr + R] -= w;
                    }
                }
            }
    // pseudo-inverse, scaled by each region's own stiffness T_R (the sum of the V-operator
    // diagonal over its nodes), so that its eigenvalues compare with those of the row-scaled
    // fine operator: the constant of an isolated conductor (coupled only through the floor)
    // lands near 1e-19 and is dropped, a body attached to others through a few edges keeps
    // its small but resolvable eigenvalue.  `cut` bounds the amplification 1/lambda to what
    // the inner vectors' precision carries.
    std::vector<double> dsq(Kr), A((size_t)Kr * Kr), Q;
    for (int r = 0; r < Kr; r++) dsq[r] = Tr[r] > 0 ? 1.0 / std::sqrt(Tr[r]) : 0.0;
    for (int r = 0; r < Kr; r++)
        for (int c = 0; c < Kr; c++) A[(size_t)r * Kr + c] = Km[(size_t)r * Kr + c] * dsq[r] * dsq[c];
    sym_eig_jacobi(Kr, A, Q);
    std::vector<double> Kpi((size_t)Kr * Kr, 0.0);
    int kept = 0;
    for (int e = 0; e < Kr; e++) {
        const double lam = A[(size_t)e * Kr + e];
        if (!(lam > cut)) continue;
        kept++;
        for (int r = 0; r < Kr; r++)
            for (int c = 0; c < Kr; c++)
                Kpi[(size_t)r * Kr + c] += Q[(size_t)r * Kr + e] * Q[(size_t)c * Kr + e] / lam;
    }
    if (kept == 0) return 0;                          // only null modes: nothing to add
    for (int r = 0; r < Kr; r++)
        for (int c = 0; c < Kr; c++) Kpi[(size_t)r * Kr + c] *= dsq[r] * dsq[c];
    // node lists, region by region
    std::vector<int> hptr(Kr + 1, 0), hrows, hrid;
    for (long long p = 0; p < Nn; p++)
        if (nreg[p] >= 0) hptr[nreg[p] + 1]++;
    for (int r = 0; r < Kr; r++) hptr[r + 1] += hptr[r];
    hrows.resize(hptr[Kr]);
    hrid.resize(hptr[Kr]);
    std::vector<int> fill(hptr.begin(), hptr.end() - 1);
    const QPL L = qms_pl(g);                        // rows in the inner solver's padded layout
    for (long long p = 0; p < Nn; p++)
        if (nreg[p] >= 0) {
            const int r = nreg[p];
            const int i = (int)(p % Nx) + 1, j = (int)((p / Nx) % Ny) + 1, k = (int)(p / ((long long)Nx * Ny)) + 1;
            hrows[fill[r]] = (int)(3 * L.comp + qms_pl_node(g, L, i, j, k));
            hrid[fill[r]] = r;
            fill[r]++;
        }
    const int total = hptr[Kr];
    std::vector<int> hcptr, hrchunk(Kr + 1);
    for (int r = 0; r < Kr; r++) {
        hrchunk[r] = (int)hcptr.size();
        for (int e = hptr[r]; e < hptr[r + 1]; e += QMS_REGION_CHUNK) hcptr.push_back(e);
    }
    hrchunk[Kr] = (int)hcptr.size();
    hcptr.push_back(total);
    const int nc = hrchunk[Kr];
    if (cudaMalloc(&cptr, (nc + 1) * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&rchunk, (Kr + 1) * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&rows, total * sizeof(int)) != cudaSuccess || cudaMalloc(&rid, total * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&Kp, (size_t)Kr * Kr * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&part, nc * sizeof(double)) != cudaSuccess || cudaMalloc(&y, Kr * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&counter, sizeof(unsigned)) != cudaSuccess) {
        err = "out of device memory (region coarse space)";
        release();
        return -1;
    }
    cudaMemsetAsync(counter, 0, sizeof(unsigned), st);
    cudaMemcpyAsync(cptr, hcptr.data(), (nc + 1) * sizeof(int), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(rchunk, hrchunk.data(), (Kr + 1) * sizeof(int), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(rows, hrows.data(), total * sizeof(int), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(rid, hrid.data(), total * sizeof(int), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(Kp, Kpi.data(), (size_t)Kr * Kr * sizeof(double), cudaMemcpyHostToDevice, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {   // the host vectors go out of scope
        err = "region coarse space upload failed";
        release();
        return -1;
    }
    K = Kr;
    nchunk = nc;
    total_entries = total;
    return 0;
}

template <typename T>
void QmsRegions::apply(const T* b, const float* bscale, T* z, cudaStream_t st, long long& launches) {
    if (K == 0) return;
    pdl_launch(qk_region_solve<T>, dim3(nchunk), dim3(256), 0, st, 0, cptr, rchunk, rows, b, bscale, part, K, Kp, y,
               counter);
    const int total = total_entries;
    pdl_launch(qk_region_scatter<T>, dim3((total + 255) / 256), dim3(256), 0, st, 0, total, rows, rid, y, z);
    launches += 2;
}
template void QmsRegions::apply<float>(const float*, const float*, float*, cudaStream_t, long long&);
template void QmsRegions::apply<double>(const double*, const float*, double*, cudaStream_t, long long&);
