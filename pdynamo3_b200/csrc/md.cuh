// Boys functions and McMurchie-Davidson (Hermite Gaussian) primitive quartets for the shell classes of
// low total angular momentum (McMurchie and Davidson, J. Comput. Phys. 26, 218 (1978); Helgaker,
// Joergensen and Olsen, Molecular Electronic-Structure Theory, chapter 9).
//
// A Gaussian product of the bra pair is expanded in Hermite Gaussians at its centre P,
//   x_A^i x_B^j exp(..) = sum_t E_t^(ij) (d/dP_x)^t exp(-p x_P^2),
// so that (ab|cd) = sum_T E_T^(ab) sum_T' (-1)^|T'| E_T'^(cd) R_(T+T'), with the Hermite Coulomb
// integrals R_tuv = (d/dP)^tuv of the prefactor times F_0(alpha |P - Q|^2).
//
// Why these classes use it instead of the Rys rule: a Rys rule of n nodes reads 2 n Chebyshev series of
// 9 to 15 coefficients, each 16-byte load of a warp touching 32 different rows, and that gather kept the
// L1 data pipe 81-92% busy in the s/p classes while the FP64 pipe ran at 25-33%.  One Boys function of
// the highest order is one run of 64 bytes (four loads); exp(-x) and the downward recursion give the
// others, and the Hermite sums take fewer operations than n_R products per component.
#pragma once
#include "common.cuh"

// Each translation unit that includes this header holds its own copy of the table (about 190 KB).
#define BOYS_TABLE_QUALIFIER static __device__ const __align__(64)
#include "boys_table.inc"
#undef BOYS_TABLE_QUALIFIER

// F_0 .. F_M at x >= 0: the table's polynomial for F_M below BOYS_XMAX, its limit above, then
// F_(m-1) = (2 x F_m + exp(-x)) / (2 m - 1), stable downwards.
template <int M>
__device__ __forceinline__ void boys(double x, double (&F)[M + 1]) {
    static_assert(M <= BOYS_MMAX, "Boys table order");
    if (x >= (double)BOYS_XMAX) {
        const double rs = rsqrt(x), rx = rs * rs;
        F[0] = 0.88622692545275801365 * rs;  // sqrt(pi) / 2
#pragma unroll
        for (int m = 1; m <= M; ++m) F[m] = F[m - 1] * (m - 0.5) * rx;
        return;
    }
    const int it = (int)(x * BOYS_INVH);
    const double t = fma(x, 2.0 * BOYS_INVH, -(2.0 * it + 1.0));
    const double2 *__restrict__ c = reinterpret_cast<const double2 *>(boys_table) + 4 * (M * (BOYS_XMAX * BOYS_INVH) + it);
    const double2 c0 = __ldg(c), c1 = __ldg(c + 1), c2 = __ldg(c + 2), c3 = __ldg(c + 3);
    const double t2 = t * t;
    const double lo = fma(fma(c1.y, t, c1.x), t2, fma(c0.y, t, c0.x));
    const double hi = fma(fma(c3.y, t, c3.x), t2, fma(c2.y, t, c2.x));
    F[M] = fma(hi, t2 * t2, lo);
    if constexpr (M > 0) {
        const double ex = exp(-x), x2 = 2.0 * x;
#pragma unroll
        for (int m = M; m > 0; --m) F[m - 1] = fma(x2, F[m], ex) * (1.0 / (2 * m - 1));
    }
}

// The same for the FP32 quartets of the mixed mode.  Two or three downward steps leave F_0 up to 2.8e-7 off
// (the weights of the single-precision Rys rule sum to it within 1.4e-7), but the Hermite sums take fewer
// operations: Fock matrices of 31 molecules of 9 to 60 atoms at the mode's cut of 1e-6 differ from FP64 ones by
// 5e-14 to 3e-13 of their norm, on average 4% less than with the Rys rule in the same kernels.  F_0, or every
// order, from a table of its own made no difference to that.
template <int M>
__device__ __forceinline__ void boys(float x, float (&F)[M + 1]) {
    static_assert(M <= BOYS_MMAX, "Boys table order");
    if (x >= (float)BOYS_XMAX) {
        const float rs = rsqrtf(x), rx = rs * rs;
        F[0] = 0.886226925f * rs;
#pragma unroll
        for (int m = 1; m <= M; ++m) F[m] = F[m - 1] * (m - 0.5f) * rx;
        return;
    }
    const int it = (int)(x * BOYSF_INVH);
    const float t = fmaf(x, 2.0f * BOYSF_INVH, -(2.0f * it + 1.0f));
    const float4 c = __ldg(reinterpret_cast<const float4 *>(boys_tablef) + M * (BOYS_XMAX * BOYSF_INVH) + it);
    F[M] = fmaf(fmaf(fmaf(c.w, t, c.z), t, c.y), t, c.x);
    if constexpr (M > 0) {
        const float ex = expf(-x), x2 = 2.0f * x;
#pragma unroll
        for (int m = M; m > 0; --m) F[m - 1] = fmaf(x2, F[m], ex) * (1.0f / (2 * m - 1));
    }
}

// Hermite indices of total order <= L in one array: by x order t, then u, then v.
__host__ __device__ constexpr int nherm(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ constexpr int hidx(int L, int t, int u, int v) {
    // after the complete planes of smaller t and the rows of smaller u
    return nherm(L) - nherm(L - t) + ((L - t + 1) * (L - t + 2) - (L - t - u + 1) * (L - t - u + 2)) / 2 + v;
}

// R_tuv, t + u + v <= L, of pref (2 pi^(5/2) / (p q sqrt(p+q)) times the contraction) at the distance
// (X, Y, Z) = P - Q and reduced exponent al = p q / (p + q).
template <int L, typename T>
__device__ __forceinline__ void hermite_coulomb(T al, T X, T Y, T Z, T pref, T (&R)[nherm(L)]) {
    T F[L + 1];
    boys<L>(al * (X * X + Y * Y + Z * Z), F);
    const T m2a = T(-2) * al;
#pragma unroll
    for (int n = 0; n <= L; ++n) {
        F[n] *= pref;
        pref *= m2a;
    }
    // from n = L down to 0: R^n to order L - n from R^(n+1) to order L - n - 1
    T a[nherm(L)], b[nherm(L)];
#pragma unroll
    for (int k = 0; k < nherm(L); ++k) a[k] = b[k] = T(0);
    a[0] = F[L];
#pragma unroll
    for (int n = L - 1; n >= 0; --n) {
#pragma unroll
        for (int t = 0; t <= L - n; ++t)
#pragma unroll
            for (int u = 0; u <= L - n - t; ++u)
#pragma unroll
                for (int v = 0; v <= L - n - t - u; ++v) {
                    T r;
                    if (t + u + v == 0) r = F[n];
                    // lower an index of one where there is one (its recursion has a single term)
                    else if (t == 1 || (t > 1 && u != 1 && v != 1))
                        r = X * a[hidx(L, t > 0 ? t - 1 : 0, u, v)] + (t > 1 ? (t - 1) * a[hidx(L, t > 1 ? t - 2 : 0, u, v)] : T(0));
                    else if (u == 1 || (u > 1 && v != 1))
                        r = Y * a[hidx(L, t, u > 0 ? u - 1 : 0, v)] + (u > 1 ? (u - 1) * a[hidx(L, t, u > 1 ? u - 2 : 0, v)] : T(0));
                    else
                        r = Z * a[hidx(L, t, u, v > 0 ? v - 1 : 0)] + (v > 1 ? (v - 1) * a[hidx(L, t, u, v > 1 ? v - 2 : 0)] : T(0));
                    b[hidx(L, t, u, v)] = r;
                }
#pragma unroll
        for (int k = 0; k < nherm(L); ++k) a[k] = b[k];
    }
#pragma unroll
    for (int k = 0; k < nherm(L); ++k) R[k] = a[k];
}

// One-dimensional Hermite coefficients E[i][j][t], t <= i + j, at the distances xa = P - A, xb = P - B with
// h = 1 / (2 p); SIGN = -1 folds the ket's (-1)^t in.
template <int LA, int LB, int SIGN, typename T>
struct Hermite1D {
    T E[LA + 1][LB + 1][LA + LB + 1];
    __device__ __forceinline__ Hermite1D(T xa, T xb, T h) {
        E[0][0][0] = T(1);
#pragma unroll
        for (int j = 0; j < LB; ++j) step(0, j, 0, j + 1, j, xb, h);
#pragma unroll
        for (int i = 0; i < LA; ++i)
#pragma unroll
            for (int j = 0; j <= LB; ++j) step(i, j, i + 1, j, i + j, xa, h);
    }
    __device__ __forceinline__ void step(int i, int j, int i1, int j1, int n, T x, T h) {
        const T sh = SIGN * h;
#pragma unroll
        for (int t = 0; t <= LA + LB; ++t) {
            if (t > n + 1) continue;
            T v = T(0);
            if (t > 0) v += sh * E[i][j][t > 0 ? t - 1 : 0];
            if (t <= n) v += x * E[i][j][t];
            if (t + 1 <= n) v += T(SIGN * (t + 1)) * E[i][j][t + 1 <= LA + LB ? t + 1 : 0];
            E[i1][j1][t] = v;
        }
    }
};

// Classes evaluated this way (the rule is explained where it is used).
__host__ __device__ constexpr bool md_class(int la, int lb, int lc, int ld) { return la + lb + lc + ld <= 3; }

// One primitive quartet added to the raw Cartesian block V[((a NB + b) NC + c) ND + d].
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void md_energy(T al, const T (&PQ)[3], T pref, const T (&PA)[3], const T (&PB)[3], T hp,
                                          const T (&QC)[3], const T (&QD)[3], T hq,
                                          T (&V)[ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD)]) {
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
    T R[nherm(L)];
    hermite_coulomb<L, T>(al, PQ[0], PQ[1], PQ[2], pref, R);
    const Hermite1D<LA, LB, 1, T> ex(PA[0], PB[0], hp), ey(PA[1], PB[1], hp), ez(PA[2], PB[2], hp);
    const Hermite1D<LC, LD, -1, T> kx(QC[0], QD[0], hq), ky(QC[1], QD[1], hq), kz(QC[2], QD[2], hq);
#pragma unroll
    for (int kc = 0; kc < NC; ++kc)
#pragma unroll
        for (int ld = 0; ld < ND; ++ld) {
            T H[nherm(LAB)];  // the bra's Hermite Gaussians with this ket component
#pragma unroll
            for (int t = 0; t <= LAB; ++t)
#pragma unroll
                for (int u = 0; u <= LAB - t; ++u)
#pragma unroll
                    for (int v = 0; v <= LAB - t - u; ++v) {
                        const int cx = cart_x(LC, kc), cy = cart_y(LC, kc), cz = cart_z(LC, kc);
                        const int dx = cart_x(LD, ld), dy = cart_y(LD, ld), dz = cart_z(LD, ld);
                        T s = T(0);
#pragma unroll
                        for (int i = 0; i <= cx + dx; ++i)
#pragma unroll
                            for (int j = 0; j <= cy + dy; ++j)
#pragma unroll
                                for (int k = 0; k <= cz + dz; ++k)
                                    s += kx.E[cx][dx][i] * ky.E[cy][dy][j] * kz.E[cz][dz][k] * R[hidx(L, t + i, u + j, v + k)];
                        H[hidx(LAB, t, u, v)] = s;
                    }
#pragma unroll
            for (int ia = 0; ia < NA; ++ia)
#pragma unroll
                for (int jb = 0; jb < NB; ++jb) {
                    const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
                    const int bx = cart_x(LB, jb), by = cart_y(LB, jb), bz = cart_z(LB, jb);
                    T s = T(0);
#pragma unroll
                    for (int i = 0; i <= ax + bx; ++i)
#pragma unroll
                        for (int j = 0; j <= ay + by; ++j)
#pragma unroll
                            for (int k = 0; k <= az + bz; ++k)
                                s += ex.E[ax][bx][i] * ey.E[ay][by][j] * ez.E[az][bz][k] * H[hidx(LAB, i, j, k)];
                    V[((ia * NB + jb) * NC + kc) * ND + ld] += s;
                }
        }
}

// Derivatives of e = sum Gam (ab|cd) of one primitive quartet: with e itself (returned), dP the gradient
// with respect to P at fixed internal geometry (that of Q is its negative), and da, db, dc, dd the
// gradients with respect to P - A, P - B, Q - C, Q - D in the Hermite coefficients.  They follow from
// sums over lowered components, d E^(ij)_t / d(P-A) = i E^(i-1,j)_t, so no integral above order L + 1 is
// formed and dP needs only the Hermite density Z_u = sum_(T+T'=u) of the quartet.
template <int LA, int LB, int LC, int LD, typename T, typename G>
__device__ __forceinline__ T md_gradient(T al, const T (&PQ)[3], T pref, const T (&PA)[3], const T (&PB)[3], T hp,
                                         const T (&QC)[3], const T (&QD)[3], T hq, const G &Gam, T (&dP)[3], T (&da)[3],
                                         T (&db)[3], T (&dc)[3], T (&dd)[3]) {
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
    T R[nherm(L + 1)];
    hermite_coulomb<L + 1, T>(al, PQ[0], PQ[1], PQ[2], pref, R);
    const Hermite1D<LA, LB, 1, T> e0(PA[0], PB[0], hp), e1(PA[1], PB[1], hp), e2(PA[2], PB[2], hp);
    const Hermite1D<LC, LD, -1, T> k0(QC[0], QD[0], hq), k1(QC[1], QD[1], hq), k2(QC[2], QD[2], hq);
    T e = T(0), Z[nherm(L)];
#pragma unroll
    for (int k = 0; k < nherm(L); ++k) Z[k] = T(0);
#pragma unroll
    for (int d = 0; d < 3; ++d) da[d] = db[d] = dc[d] = dd[d] = T(0);
    // bra components with the ket contracted
#pragma unroll
    for (int ia = 0; ia < NA; ++ia)
#pragma unroll
        for (int jb = 0; jb < NB; ++jb) {
            const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
            const int bx = cart_x(LB, jb), by = cart_y(LB, jb), bz = cart_z(LB, jb);
            T g[nherm(LCD)];
#pragma unroll
            for (int k = 0; k < nherm(LCD); ++k) g[k] = T(0);
#pragma unroll
            for (int kc = 0; kc < NC; ++kc)
#pragma unroll
                for (int ld = 0; ld < ND; ++ld) {
                    const int cx = cart_x(LC, kc), cy = cart_y(LC, kc), cz = cart_z(LC, kc);
                    const int dx = cart_x(LD, ld), dy = cart_y(LD, ld), dz = cart_z(LD, ld);
                    const T gm = T(Gam[((ia * NB + jb) * NC + kc) * ND + ld]);
#pragma unroll
                    for (int i = 0; i <= cx + dx; ++i)
#pragma unroll
                        for (int j = 0; j <= cy + dy; ++j)
#pragma unroll
                            for (int k = 0; k <= cz + dz; ++k)
                                g[hidx(LCD, i, j, k)] += gm * (k0.E[cx][dx][i] * k1.E[cy][dy][j] * k2.E[cz][dz][k]);
                }
            // Hermite density, and the potentials M_T = sum_T' g_T' R_(T+T') of this component
#pragma unroll
            for (int t = 0; t <= ax + bx; ++t)
#pragma unroll
                for (int u = 0; u <= ay + by; ++u)
#pragma unroll
                    for (int v = 0; v <= az + bz; ++v) {
                        const T E = e0.E[ax][bx][t] * e1.E[ay][by][u] * e2.E[az][bz][v];
                        T M = T(0);
#pragma unroll
                        for (int i = 0; i <= LCD; ++i)
#pragma unroll
                            for (int j = 0; j <= LCD - i; ++j)
#pragma unroll
                                for (int k = 0; k <= LCD - i - j; ++k) {
                                    const T gk = g[hidx(LCD, i, j, k)];
                                    Z[hidx(L, t + i, u + j, v + k)] += E * gk;
                                    if (t + u + v < LAB) M += gk * R[hidx(L + 1, t + i, u + j, v + k)];
                                }
                        if (t + u + v < LAB) {
                            if (ax > 0 && t < ax + bx) da[0] += T(ax) * (e0.E[ax > 0 ? ax - 1 : 0][bx][t] * e1.E[ay][by][u] * e2.E[az][bz][v]) * M;
                            if (ay > 0 && u < ay + by) da[1] += T(ay) * (e0.E[ax][bx][t] * e1.E[ay > 0 ? ay - 1 : 0][by][u] * e2.E[az][bz][v]) * M;
                            if (az > 0 && v < az + bz) da[2] += T(az) * (e0.E[ax][bx][t] * e1.E[ay][by][u] * e2.E[az > 0 ? az - 1 : 0][bz][v]) * M;
                            if (bx > 0 && t < ax + bx) db[0] += T(bx) * (e0.E[ax][bx > 0 ? bx - 1 : 0][t] * e1.E[ay][by][u] * e2.E[az][bz][v]) * M;
                            if (by > 0 && u < ay + by) db[1] += T(by) * (e0.E[ax][bx][t] * e1.E[ay][by > 0 ? by - 1 : 0][u] * e2.E[az][bz][v]) * M;
                            if (bz > 0 && v < az + bz) db[2] += T(bz) * (e0.E[ax][bx][t] * e1.E[ay][by][u] * e2.E[az][bz > 0 ? bz - 1 : 0][v]) * M;
                        }
                    }
        }
    // ket components with the bra contracted: only the lowered sums
    if constexpr (LCD > 0) {
#pragma unroll
        for (int kc = 0; kc < NC; ++kc)
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) {
                const int cx = cart_x(LC, kc), cy = cart_y(LC, kc), cz = cart_z(LC, kc);
                const int dx = cart_x(LD, ld), dy = cart_y(LD, ld), dz = cart_z(LD, ld);
                T g[nherm(LAB)];
#pragma unroll
                for (int k = 0; k < nherm(LAB); ++k) g[k] = T(0);
#pragma unroll
                for (int ia = 0; ia < NA; ++ia)
#pragma unroll
                    for (int jb = 0; jb < NB; ++jb) {
                        const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
                        const int bx = cart_x(LB, jb), by = cart_y(LB, jb), bz = cart_z(LB, jb);
                        const T gm = T(Gam[((ia * NB + jb) * NC + kc) * ND + ld]);
#pragma unroll
                        for (int i = 0; i <= ax + bx; ++i)
#pragma unroll
                            for (int j = 0; j <= ay + by; ++j)
#pragma unroll
                                for (int k = 0; k <= az + bz; ++k)
                                    g[hidx(LAB, i, j, k)] += gm * (e0.E[ax][bx][i] * e1.E[ay][by][j] * e2.E[az][bz][k]);
                    }
#pragma unroll
                for (int t = 0; t <= cx + dx; ++t)
#pragma unroll
                    for (int u = 0; u <= cy + dy; ++u)
#pragma unroll
                        for (int v = 0; v <= cz + dz; ++v) {
                            if (t + u + v >= LCD) continue;
                            T M = T(0);
#pragma unroll
                            for (int i = 0; i <= LAB; ++i)
#pragma unroll
                                for (int j = 0; j <= LAB - i; ++j)
#pragma unroll
                                    for (int k = 0; k <= LAB - i - j; ++k)
                                        M += g[hidx(LAB, i, j, k)] * R[hidx(L + 1, t + i, u + j, v + k)];
                            if (cx > 0 && t < cx + dx) dc[0] += T(cx) * (k0.E[cx > 0 ? cx - 1 : 0][dx][t] * k1.E[cy][dy][u] * k2.E[cz][dz][v]) * M;
                            if (cy > 0 && u < cy + dy) dc[1] += T(cy) * (k0.E[cx][dx][t] * k1.E[cy > 0 ? cy - 1 : 0][dy][u] * k2.E[cz][dz][v]) * M;
                            if (cz > 0 && v < cz + dz) dc[2] += T(cz) * (k0.E[cx][dx][t] * k1.E[cy][dy][u] * k2.E[cz > 0 ? cz - 1 : 0][dz][v]) * M;
                            if (dx > 0 && t < cx + dx) dd[0] += T(dx) * (k0.E[cx][dx > 0 ? dx - 1 : 0][t] * k1.E[cy][dy][u] * k2.E[cz][dz][v]) * M;
                            if (dy > 0 && u < cy + dy) dd[1] += T(dy) * (k0.E[cx][dx][t] * k1.E[cy][dy > 0 ? dy - 1 : 0][u] * k2.E[cz][dz][v]) * M;
                            if (dz > 0 && v < cz + dz) dd[2] += T(dz) * (k0.E[cx][dx][t] * k1.E[cy][dy][u] * k2.E[cz][dz > 0 ? dz - 1 : 0][v]) * M;
                        }
            }
    }
    dP[0] = dP[1] = dP[2] = T(0);
#pragma unroll
    for (int t = 0; t <= L; ++t)
#pragma unroll
        for (int u = 0; u <= L - t; ++u)
#pragma unroll
            for (int v = 0; v <= L - t - u; ++v) {
                const T z = Z[hidx(L, t, u, v)];
                e += z * R[hidx(L + 1, t, u, v)];
                dP[0] += z * R[hidx(L + 1, t + 1, u, v)];
                dP[1] += z * R[hidx(L + 1, t, u + 1, v)];
                dP[2] += z * R[hidx(L + 1, t, u, v + 1)];
            }
    return e;
}
