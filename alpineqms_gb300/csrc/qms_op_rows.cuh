// qms_op_rows.cuh -- the rows of the Yee A-V operator at one node (the same entries as the
// assembled CSR: F:476-607, F:650-781, F:824-955, F:1014-1285 and the transient additions
// F:1475-1504, F:1624-1681, F:1772-1857, F:1925-2126), shared by the stencil kernels.
//
// Each row is evaluated in difference form: every coupling pair acts on a difference of
// unknowns, so rounding scales with the variation of x rather than with x itself.
//   xs(q, dk, dj, di): unknown block q at (i + di, j + dj, k + dk), dk in {-1, 0, 1}
//   cf(q, dk, dj, di): node coefficient q (1/mu_x,y,z, sigma_x,y,z) at (i + di, j + dj, k + dk),
//                      dk in {-1, 0}
//   emit(row, acc, diag, is_a, x_row, fixed, tacc, tdiag): the row's value M x, its diagonal, its own unknown and
//                      whether it is a Dirichlet row (value and diagonal then without units); what the
//                      terms in 1 / dt add to value and diagonal where they come apart (QROW_TIME), else zero
// fij*/kf*: the (i, j) and k parts of the Dirichlet predicates qFixX/Y/Z/V.
// UNI: QROW_UNIT, cubic cells (dx = dy = dz), everything in units of 1 / h^2: P is then qms_unit_par's (1/dt,
// 1/h and the advection factors times h^2), the links' 1 / h^2 is one and left out of the products at compile
// time, and acc and diag come in those units.  A row's products fall by about a third (the kernels over
// these rows are bound by instruction issue).  QROW_TIME, the same with the terms in 1 / dt apart and in
// their own units: 1 / dt times h^2 is a rounding that a residual b - M x enlarges where sigma x / dt and b
// nearly cancel.
// VM: which velocity components may be nonzero (bit 0 x, 1 y, 2 z; 0 = no advection term);
// the terms of components outside VM are left out at compile time (they are exact zeros).
#pragma once
#include "qms_common.cuh"

enum QRowUnits { QROW_PLAIN = 0, QROW_UNIT = 1, QROW_TIME = 2 };

template <typename T>
static inline QStepPar<T> qms_unit_par(const QGrid& g, QStepPar<T> p, QRowUnits uni = QROW_UNIT) {
    if (uni == QROW_TIME) {
        p.idtx = (T)((double)p.idt / g.dx);
    } else {
        p.idtx = (T)((double)p.idt * g.dx);
        p.idt = (T)((double)p.idt * (g.dx * g.dx));
    }
    p.idx2 = p.idy2 = p.idz2 = p.idxdy = p.idxdz = p.idydz = T(1);
    p.i2dx = p.i2dy = p.i2dz = (T)(0.5 * g.dx);
    p.idx = p.idy = p.idz = (T)g.dx;
    p.i2dx2 = p.i2dy2 = p.i2dz2 = p.i2dxdy = p.i2dxdz = p.i2dydz = T(0.5);
    return p;
}
template <typename T, int VM, int UNI = QROW_PLAIN, typename XS, typename CF, typename EMIT>
__device__ __forceinline__ void qms_op_node(const QGrid& g, const QStepPar<T>& P, int i, int j, int k, bool fijX,
                                            bool fijY, bool fijZ, bool kfA, bool kfZ, long long rX, long long rY,
                                            long long rZ, long long rV, XS xs, CF cf, EMIT emit) {
        auto lk = [](T c, T w) -> T { if constexpr (UNI) return c; else return c * w; };   // a link times its 1 / h^2
        // a row's sum t and its term m in 1 / dt, together or (QROW_TIME) apart
        auto with = [](T m, T t) -> T { if constexpr (UNI == QROW_TIME) return t; else return m + t; };
        auto apart = [](T m) -> T { if constexpr (UNI == QROW_TIME) return m; else return T(0); };
        constexpr bool HX = (VM & 1) != 0, HY = (VM & 2) != 0, HZ = (VM & 4) != 0;
        // ---------------------------------------------------------------- Ax
        if (i <= g.xs) {
            const long long row = rX;
            if (fijX || kfA) {
                emit(row, xs(0, 0, 0, 0), T(1), true, xs(0, 0, 0, 0), true, T(0), T(0));
            } else {
                const T s = cf(3, 0, 0, 0);
                const T my_km = cf(1, -1, 0, 0), my_k = cf(1, 0, 0, 0);
                const T mz_jm = cf(2, 0, -1, 0), mz_j = cf(2, 0, 0, 0);
                const T mx_im = cf(0, 0, 0, -1), mx_i = cf(0, 0, 0, 0);
                const T svy = HY ? s * P.vy : T(0), svz = HZ ? s * P.vz : T(0);
                const T d = lk(mz_j + mz_jm, P.idy2) + lk(my_k + my_km, P.idz2) + lk(mx_i + mx_im, P.idx2);
                // difference form: every coupling pair is applied to a difference of unknowns,
                // so the rounding error scales with the variation of x, not with x itself
                const T X0 = xs(0, 0, 0, 0);
                const T mass = s * P.idt, tacc = mass * X0;
                T acc = with(tacc, lk(my_km, P.idz2) * (X0 - xs(0, -1, 0, 0)) + lk(my_k, P.idz2) * (X0 - xs(0, 1, 0, 0)));
                acc += lk(mz_jm, P.idy2) * (X0 - xs(0, 0, -1, 0)) + lk(mz_j, P.idy2) * (X0 - xs(0, 0, 1, 0));
                acc += lk(mx_im, P.idx2) * (X0 - xs(0, 0, 0, -1)) + lk(mx_i, P.idx2) * (X0 - xs(0, 0, 0, 1));
                if constexpr (HZ) acc += svz * P.i2dz * (xs(0, -1, 0, 0) - xs(0, 1, 0, 0));
                if constexpr (HY) acc += svy * P.i2dy * (xs(0, 0, -1, 0) - xs(0, 0, 1, 0));
                acc += (HY ? lk(mz_jm, P.idxdy) - svy * P.i2dx : lk(mz_jm, P.idxdy)) * (xs(1, 0, -1, 0) - xs(1, 0, -1, 1));
                acc += (HY ? lk(mz_j, P.idxdy) + svy * P.i2dx : lk(mz_j, P.idxdy)) * (xs(1, 0, 0, 1) - xs(1, 0, 0, 0));
                acc += (HZ ? lk(my_km, P.idxdz) - svz * P.i2dx : lk(my_km, P.idxdz)) * (xs(2, -1, 0, 0) - xs(2, -1, 0, 1));
                acc += (HZ ? lk(my_k, P.idxdz) + svz * P.i2dx : lk(my_k, P.idxdz)) * (xs(2, 0, 0, 1) - xs(2, 0, 0, 0));
                acc += s * P.idx * (xs(3, 0, 0, 1) - xs(3, 0, 0, 0));
                emit(row, acc, with(mass, d), true, xs(0, 0, 0, 0), false, apart(tacc), apart(mass));
            }
        }
        // ---------------------------------------------------------------- Ay
        if (j <= g.ys) {
            const long long row = rY;
            if (fijY || kfA) {
                emit(row, xs(1, 0, 0, 0), T(1), true, xs(1, 0, 0, 0), true, T(0), T(0));
            } else {
                const T s = cf(4, 0, 0, 0);
                const T mz_im = cf(2, 0, 0, -1), mz_i = cf(2, 0, 0, 0);
                const T mx_km = cf(0, -1, 0, 0), mx_k = cf(0, 0, 0, 0);
                const T my_jm = cf(1, 0, -1, 0), my_j = cf(1, 0, 0, 0);
                const T svx = HX ? s * P.vx : T(0), svz = HZ ? s * P.vz : T(0);
                const T d = lk(mz_i + mz_im, P.idx2) + lk(mx_k + mx_km, P.idz2) + lk(my_j + my_jm, P.idy2);
                const T Y0 = xs(1, 0, 0, 0);
                const T mass = s * P.idt, tacc = mass * Y0;
                T acc = with(tacc, lk(mx_km, P.idz2) * (Y0 - xs(1, -1, 0, 0)) + lk(mx_k, P.idz2) * (Y0 - xs(1, 1, 0, 0)));
                acc += lk(my_jm, P.idy2) * (Y0 - xs(1, 0, -1, 0)) + lk(my_j, P.idy2) * (Y0 - xs(1, 0, 1, 0));
                acc += lk(mz_im, P.idx2) * (Y0 - xs(1, 0, 0, -1)) + lk(mz_i, P.idx2) * (Y0 - xs(1, 0, 0, 1));
                if constexpr (HZ) acc += svz * P.i2dz * (xs(1, -1, 0, 0) - xs(1, 1, 0, 0));
                if constexpr (HX) acc += svx * P.i2dx * (xs(1, 0, 0, -1) - xs(1, 0, 0, 1));
                acc += (HX ? lk(mz_im, P.idxdy) - svx * P.i2dy : lk(mz_im, P.idxdy)) * (xs(0, 0, 0, -1) - xs(0, 0, 1, -1));
                acc += (HX ? lk(mz_i, P.idxdy) + svx * P.i2dy : lk(mz_i, P.idxdy)) * (xs(0, 0, 1, 0) - xs(0, 0, 0, 0));
                acc += (HZ ? lk(mx_km, P.idydz) - svz * P.i2dy : lk(mx_km, P.idydz)) * (xs(2, -1, 0, 0) - xs(2, -1, 1, 0));
                acc += (HZ ? lk(mx_k, P.idydz) + svz * P.i2dy : lk(mx_k, P.idydz)) * (xs(2, 0, 1, 0) - xs(2, 0, 0, 0));
                acc += s * P.idy * (xs(3, 0, 1, 0) - xs(3, 0, 0, 0));
                emit(row, acc, with(mass, d), true, xs(1, 0, 0, 0), false, apart(tacc), apart(mass));
            }
        }
        // ---------------------------------------------------------------- Az
        if (k <= g.zs) {
            const long long row = rZ;
            if (fijZ || kfZ) {
                emit(row, xs(2, 0, 0, 0), T(1), true, xs(2, 0, 0, 0), true, T(0), T(0));
            } else {
                const T s = cf(5, 0, 0, 0);
                const T my_im = cf(1, 0, 0, -1), my_i = cf(1, 0, 0, 0);
                const T mx_jm = cf(0, 0, -1, 0), mx_j = cf(0, 0, 0, 0);
                const T mz_km = cf(2, -1, 0, 0), mz_k = cf(2, 0, 0, 0);
                const T svx = HX ? s * P.vx : T(0), svy = HY ? s * P.vy : T(0);
                const T d = lk(my_i + my_im, P.idx2) + lk(mx_j + mx_jm, P.idy2) + lk(mz_k + mz_km, P.idz2);
                const T Z0 = xs(2, 0, 0, 0);
                const T mass = s * P.idt, tacc = mass * Z0;
                T acc = with(tacc, lk(mz_km, P.idz2) * (Z0 - xs(2, -1, 0, 0)) + lk(mz_k, P.idz2) * (Z0 - xs(2, 1, 0, 0)));
                acc += lk(mx_jm, P.idy2) * (Z0 - xs(2, 0, -1, 0)) + lk(mx_j, P.idy2) * (Z0 - xs(2, 0, 1, 0));
                acc += lk(my_im, P.idx2) * (Z0 - xs(2, 0, 0, -1)) + lk(my_i, P.idx2) * (Z0 - xs(2, 0, 0, 1));
                if constexpr (HY) acc += svy * P.i2dy * (xs(2, 0, -1, 0) - xs(2, 0, 1, 0));
                if constexpr (HX) acc += svx * P.i2dx * (xs(2, 0, 0, -1) - xs(2, 0, 0, 1));
                acc += (HX ? lk(my_im, P.idxdz) - svx * P.i2dz : lk(my_im, P.idxdz)) * (xs(0, 0, 0, -1) - xs(0, 1, 0, -1));
                acc += (HX ? lk(my_i, P.idxdz) + svx * P.i2dz : lk(my_i, P.idxdz)) * (xs(0, 1, 0, 0) - xs(0, 0, 0, 0));
                acc += (HY ? lk(mx_jm, P.idydz) - svy * P.i2dz : lk(mx_jm, P.idydz)) * (xs(1, 0, -1, 0) - xs(1, 1, -1, 0));
                acc += (HY ? lk(mx_j, P.idydz) + svy * P.i2dz : lk(mx_j, P.idydz)) * (xs(1, 1, 0, 0) - xs(1, 0, 0, 0));
                acc += s * P.idz * (xs(3, 1, 0, 0) - xs(3, 0, 0, 0));
                emit(row, acc, with(mass, d), true, xs(2, 0, 0, 0), false, apart(tacc), apart(mass));
            }
        }
        // ---------------------------------------------------------------- V
        {
            const long long row = rV;
            if (fijZ || kfA) {
                emit(row, xs(3, 0, 0, 0), T(1), false, xs(3, 0, 0, 0), true, T(0), T(0));
            } else {
                const T sx0 = cf(3, 0, 0, 0), sx1 = cf(3, 0, 0, -1);
                const T sy0 = cf(4, 0, 0, 0), sy1 = cf(4, 0, -1, 0);
                const T sz0 = cf(5, 0, 0, 0), sz1 = cf(5, -1, 0, 0);
                const T fx0 = fmax(sx0, P.sigfloor), fx1 = fmax(sx1, P.sigfloor);
                const T fy0 = fmax(sy0, P.sigfloor), fy1 = fmax(sy1, P.sigfloor);
                const T fz0 = fmax(sz0, P.sigfloor), fz1 = fmax(sz1, P.sigfloor);
                const T d = lk(fx0 + fx1, P.idx2) + lk(fy0 + fy1, P.idy2) + lk(fz0 + fz1, P.idz2);
                const T V0 = xs(3, 0, 0, 0);
                T acc = lk(fz1, P.idz2) * (V0 - xs(3, -1, 0, 0)) + lk(fz0, P.idz2) * (V0 - xs(3, 1, 0, 0));
                acc += lk(fy1, P.idy2) * (V0 - xs(3, 0, -1, 0)) + lk(fy0, P.idy2) * (V0 - xs(3, 0, 1, 0));
                acc += lk(fx1, P.idx2) * (V0 - xs(3, 0, 0, -1)) + lk(fx0, P.idx2) * (V0 - xs(3, 0, 0, 1));
                const T axm = xs(0, 0, 0, -1), ax0 = xs(0, 0, 0, 0);
                const T aym = xs(1, 0, -1, 0), ay0 = xs(1, 0, 0, 0);
                const T azm = xs(2, -1, 0, 0), az0 = xs(2, 0, 0, 0);
                // div(sigma A) / dt: s0 a0 - s1 a1 = s0 (a0 - a1) + (s0 - s1) a1 (exact inside a body)
                const T jx = sx0 * (ax0 - axm) + (sx0 - sx1) * axm, jy = sy0 * (ay0 - aym) + (sy0 - sy1) * aym;
                const T jz = sz0 * (az0 - azm) + (sz0 - sz1) * azm;
                const T tacc = UNI ? P.idtx * (jx + jy + jz) : T(0);
                if constexpr (UNI) acc = with(tacc, acc);
                else acc += P.idt * (jx * P.idx + jy * P.idy + jz * P.idz);
                // div(sigma v x curl A), grouped by velocity component into differences
                const T vx = P.vx, vy = P.vy, vz = P.vz;
                // Ax neighbours
                const T SA = axm + ax0;
                if constexpr (HZ)
                    acc += vz * P.i2dxdz * (sx1 * (xs(0, -1, 0, -1) - xs(0, 1, 0, -1)) +
                                             sx0 * (xs(0, 1, 0, 0) - xs(0, -1, 0, 0)));
                if constexpr (HY)
                    acc += vy * P.i2dxdy * (sx1 * (xs(0, 0, -1, -1) - xs(0, 0, 1, -1)) +
                                             sx0 * (xs(0, 0, 1, 0) - xs(0, 0, -1, 0)));
                if constexpr (HX) {
                    acc += vx * P.i2dy2 * (sy1 * (SA - (xs(0, 0, -1, -1) + xs(0, 0, -1, 0))) +
                                           sy0 * (SA - (xs(0, 0, 1, -1) + xs(0, 0, 1, 0))));
                    acc += vx * P.i2dz2 * (sz1 * (SA - (xs(0, -1, 0, -1) + xs(0, -1, 0, 0))) +
                                           sz0 * (SA - (xs(0, 1, 0, -1) + xs(0, 1, 0, 0))));
                }
                // Ay neighbours
                const T SB = aym + ay0;
                if constexpr (HZ)
                    acc += vz * P.i2dydz * (sy1 * (xs(1, -1, -1, 0) - xs(1, 1, -1, 0)) +
                                             sy0 * (xs(1, 1, 0, 0) - xs(1, -1, 0, 0)));
                if constexpr (HX)
                    acc += vx * P.i2dxdy * (sy1 * (xs(1, 0, -1, -1) - xs(1, 0, -1, 1)) +
                                             sy0 * (xs(1, 0, 0, 1) - xs(1, 0, 0, -1)));
                if constexpr (HY) {
                    acc += vy * P.i2dx2 * (sx1 * (SB - (xs(1, 0, -1, -1) + xs(1, 0, 0, -1))) +
                                           sx0 * (SB - (xs(1, 0, -1, 1) + xs(1, 0, 0, 1))));
                    acc += vy * P.i2dz2 * (sz1 * (SB - (xs(1, -1, -1, 0) + xs(1, -1, 0, 0))) +
                                           sz0 * (SB - (xs(1, 1, -1, 0) + xs(1, 1, 0, 0))));
                }
                // Az neighbours
                const T SC = azm + az0;
                if constexpr (HY)
                    acc += vy * P.i2dydz * (sz1 * (xs(2, -1, -1, 0) - xs(2, -1, 1, 0)) +
                                             sz0 * (xs(2, 0, 1, 0) - xs(2, 0, -1, 0)));
                if constexpr (HX)
                    acc += vx * P.i2dxdz * (sz1 * (xs(2, -1, 0, -1) - xs(2, -1, 0, 1)) +
                                             sz0 * (xs(2, 0, 0, 1) - xs(2, 0, 0, -1)));
                if constexpr (HZ) {
                    acc += vz * P.i2dx2 * (sx1 * (SC - (xs(2, -1, 0, -1) + xs(2, 0, 0, -1))) +
                                           sx0 * (SC - (xs(2, -1, 0, 1) + xs(2, 0, 0, 1))));
                    acc += vz * P.i2dy2 * (sy1 * (SC - (xs(2, -1, -1, 0) + xs(2, 0, -1, 0))) +
                                           sy0 * (SC - (xs(2, -1, 1, 0) + xs(2, 0, 1, 0))));
                }
                emit(row, acc, d, false, xs(3, 0, 0, 0), false, apart(tacc), T(0));
            }
        }
}
