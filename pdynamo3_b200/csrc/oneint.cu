// One-electron integrals (overlap, kinetic, electron-nuclear) and their gradients.
//
// Replaces GaussianBasisContainerIntegrals_f1KOf1i / _f1KOf1R1
// (GaussianBases/__extensions__/csource/GaussianBasisContainerIntegrals_f1Xg1.c:233,298) and
// _f2Cm1V / _f2Cm1R1 (GaussianBasisContainerIntegrals_f2Cp1.c:104,30).  One warp per shell
// pair; overlap and kinetic by the Obara-Saika recursion, electron-nuclear attraction by Boys
// functions and Hermite sums with the nucleus as a narrow Gaussian charge, as the reference models it.
// Raw Cartesian integrals; the per-component normalisation is applied by the caller (N S N).
#include "context.h"
#include "md.cuh"

namespace {

constexpr double PI = 3.141592653589793;
// Nuclei are normalised Gaussian charges of width 1e-4 bohr, exponent 4/(w^2 pi)
// (GaussianBases/__extensions__/cinclude/GaussianNucleus.h:13-15).  NUC_PREF =
// 2 pi^(5/2) (zeta/pi)^(3/2) / zeta, so that V = -Z NUC_PREF/(p sqrt(p+zeta)) K sum w Ix Iy Iz.
constexpr double NUC_ZETA = 4.0 / (1.0e-4 * 1.0e-4 * PI);
#define NUC_PREF (34.986836655249725 * sqrt(NUC_ZETA / PI) / PI)

// 1D overlap table S[i][j], i <= IM, j <= JM, without the exponential prefactor.
template <int IM, int JM>
__device__ __forceinline__ void os_overlap(double (&S)[IM + 1][JM + 1], double PA, double PB, double r2p) {
    S[0][0] = 1.0;
#pragma unroll
    for (int i = 0; i < IM; ++i) S[i + 1][0] = PA * S[i][0] + (i > 0 ? i * r2p * S[i > 0 ? i - 1 : 0][0] : 0.0);
#pragma unroll
    for (int j = 0; j < JM; ++j)
#pragma unroll
        for (int i = 0; i <= IM; ++i)
            S[i][j + 1] = PB * S[i][j] + (i > 0 ? i * r2p * S[i > 0 ? i - 1 : 0][j] : 0.0) +
                          (j > 0 ? j * r2p * S[i][j > 0 ? j - 1 : 0] : 0.0);
}

// 1D kinetic piece: -1/2 d^2/dx^2 acting on the second function, x^j exp(-b x^2).
template <int IM, int JM>
__device__ __forceinline__ double kin1d(const double (&S)[IM + 1][JM + 1], int i, int j, double b) {
    double t = -2.0 * b * (2 * j + 1) * S[i][j] + 4.0 * b * b * S[i][j + 2 <= JM ? j + 2 : JM];
    if (j >= 2) t += j * (j - 1) * S[i][j >= 2 ? j - 2 : 0];
    return -0.5 * t;
}

__device__ __forceinline__ void sh_xyz(const DeviceBasis &bs, int sh, double *r) {
    const int at = bs.sh_atom[sh];
    r[0] = bs.atom_xyz[3 * at]; r[1] = bs.atom_xyz[3 * at + 1]; r[2] = bs.atom_xyz[3 * at + 2];
}

// One warp per shell pair: its lanes take the (primitive, nucleus) terms of the attraction in turn (and the
// primitives of overlap and kinetic energy), so that the few contracted s pairs (up to 36 primitives times
// all nuclei, each a Boys function) do not run in one thread.  A nucleus is the ket (C|C) with one s
// function: the Hermite sums of md.cuh with an empty ket side.  With one thread per pair and Rys rules, 96
// atoms (25,000 s pairs: five warps per SM) took 0.89 ms for the (s|s) class,
// 2.2 ms for all; now 0.09 ms, and 0.13 ms for the longest, (d|d).
constexpr int OPB = 4;  // pairs (warps) per block

template <int N>
__device__ __forceinline__ void store_pair(const double (&v)[N], int nb, int oa, int ob, int n, double *__restrict__ M) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int f = 0; f < N; ++f) {
        const double t = warp_sum(v[f]);
        const int ia = f / nb, jb = f % nb;
        if (lane == 0) { M[(oa + ia) * n + ob + jb] = t; M[(ob + jb) * n + oa + ia] = t; }
    }
}

template <int LA, int LB>
__global__ void __launch_bounds__(32 * OPB) oneint_kernel(PairList pl, PrimPairs pp, DeviceBasis bs, int n,
                                                          double *__restrict__ Sm, double *__restrict__ Tm,
                                                          double *__restrict__ Vm) {
    const int t = blockIdx.x * OPB + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= pl.n) return;
    constexpr int NA = ncart(LA), NB = ncart(LB);
    const int A = pl.shA[t], B = pl.shB[t];
    double rA[3], rB[3];
    sh_xyz(bs, A, rA);
    sh_xyz(bs, B, rB);
    const int oa = bs.sh_bf[A], ob = bs.sh_bf[B];
    const int p0 = pl.poff[t], np = pl.np[t];
    {
        double s[NA * NB], k[NA * NB];
#pragma unroll
        for (int i = 0; i < NA * NB; ++i) { s[i] = 0.0; k[i] = 0.0; }
        for (int ip = p0 + lane; ip < p0 + np; ip += 32) {
            const double b = pp.b[ip], p = pp.a[ip] + b, r2p = 0.5 / p;
            const double P[3] = {pp.Px[ip], pp.Py[ip], pp.Pz[ip]};
            double Sx[LA + 1][LB + 3], Sy[LA + 1][LB + 3], Sz[LA + 1][LB + 3];
            os_overlap<LA, LB + 2>(Sx, P[0] - rA[0], P[0] - rB[0], r2p);
            os_overlap<LA, LB + 2>(Sy, P[1] - rA[1], P[1] - rB[1], r2p);
            os_overlap<LA, LB + 2>(Sz, P[2] - rA[2], P[2] - rB[2], r2p);
            const double sp = PI / p;
            const double pref = sp * sqrt(sp) * pp.K[ip];
#pragma unroll
            for (int ia = 0; ia < NA; ++ia)
#pragma unroll
                for (int jb = 0; jb < NB; ++jb) {
                    const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
                    const int bx = cart_x(LB, jb), by = cart_y(LB, jb), bz = cart_z(LB, jb);
                    const double ox = Sx[ax][bx], oy = Sy[ay][by], oz = Sz[az][bz];
                    s[ia * NB + jb] += pref * ox * oy * oz;
                    k[ia * NB + jb] += pref * (kin1d<LA, LB + 2>(Sx, ax, bx, b) * oy * oz + ox * kin1d<LA, LB + 2>(Sy, ay, by, b) * oz +
                                               ox * oy * kin1d<LA, LB + 2>(Sz, az, bz, b));
                }
        }
        store_pair<NA * NB>(s, NB, oa, ob, n, Sm);
        store_pair<NA * NB>(k, NB, oa, ob, n, Tm);
    }
    // electron-nuclear attraction with Gaussian nuclei: -sum_C Z_C (ab|C) with the nucleus a normalised
    // Gaussian of exponent NUC_ZETA, i.e. a (ab|ss) integral with q = NUC_ZETA
    double v[NA * NB];
#pragma unroll
    for (int i = 0; i < NA * NB; ++i) v[i] = 0.0;
    const double zero[3] = {0.0, 0.0, 0.0};
    for (int idx = lane; idx < np * bs.natom; idx += 32) {
        const int j = idx / bs.natom, c = idx - j * bs.natom, ip = p0 + j;
        const double Z = bs.atom_Z[c];
        if (Z == 0.0) continue;
        const double p = pp.a[ip] + pp.b[ip], rs = rsqrt(p + NUC_ZETA);
        const double P[3] = {pp.Px[ip], pp.Py[ip], pp.Pz[ip]};
        const double PA[3] = {P[0] - rA[0], P[1] - rA[1], P[2] - rA[2]}, PB[3] = {P[0] - rB[0], P[1] - rB[1], P[2] - rB[2]};
        const double PC[3] = {P[0] - bs.atom_xyz[3 * c], P[1] - bs.atom_xyz[3 * c + 1], P[2] - bs.atom_xyz[3 * c + 2]};
        md_energy<LA, LB, 0, 0, double>(p * NUC_ZETA * rs * rs, PC, -Z * NUC_PREF * rs * pp.Kp[ip], PA, PB, pp.hp[ip], zero,
                                        zero, 0.0, v);
    }
    store_pair<NA * NB>(v, NB, oa, ob, n, Vm);
}

// Gradient of sum_uv [P_uv (T+V)_uv - Ws_uv S_uv] with respect to nuclear positions, where
// P and Ws carry the component normalisation (N P N).  Ws is the energy-weighted density
// sum_i n_i e_i C C^T.
//
// One warp per shell pair as above; lanes take nuclei (the smallest power of two above natom of them, up to
// 32, the rest of the warp further primitives), so that the term on a nucleus leaves once per pair and not
// once per primitive, and lanes add to different elements.  The blocks add to partial arrays (pdg_grad_copy).
// One thread per pair, with three atomics per primitive and nucleus of which all lanes met on one address:
// 2.1 ms of a 42-atom gradient, 0.35 ms of that of 2 waters.
template <int LA, int LB>
__global__ void __launch_bounds__(32 * OPB) oneint_grad_kernel(PairList pl, PrimPairs pp, DeviceBasis bs, int n,
                                                               const double *__restrict__ Pm, const double *__restrict__ Wm,
                                                               double *__restrict__ part, int gstride) {
    const int t = blockIdx.x * OPB + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= pl.n) return;
    constexpr int NA = ncart(LA), NB = ncart(LB);
    double *__restrict__ grad = pdg_grad_copy(part, gstride);
    const int A = pl.shA[t], B = pl.shB[t];
    const int atA = bs.sh_atom[A], atB = bs.sh_atom[B];
    double rA[3], rB[3];
    sh_xyz(bs, A, rA);
    sh_xyz(bs, B, rB);
    const int oa = bs.sh_bf[A], ob = bs.sh_bf[B];
    const double fac = (A == B) ? 1.0 : 2.0;
    const int p0 = pl.poff[t], np = pl.np[t];
    double Pab[NA * NB];
#pragma unroll
    for (int ia = 0; ia < NA; ++ia)
#pragma unroll
        for (int jb = 0; jb < NB; ++jb) Pab[ia * NB + jb] = fac * Pm[(oa + ia) * n + ob + jb];
    double gA[3] = {0.0, 0.0, 0.0}, gB[3] = {0.0, 0.0, 0.0};
    if (atA != atB) {
        double Wab[NA * NB];
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
            for (int jb = 0; jb < NB; ++jb) Wab[ia * NB + jb] = fac * Wm[(oa + ia) * n + ob + jb];
        for (int ip = p0 + lane; ip < p0 + np; ip += 32) {
            const double a = pp.a[ip], b = pp.b[ip], p = a + b, r2p = 0.5 / p;
            const double P[3] = {pp.Px[ip], pp.Py[ip], pp.Pz[ip]};
            double Sx[LA + 2][LB + 3], Sy[LA + 2][LB + 3], Sz[LA + 2][LB + 3];
            os_overlap<LA + 1, LB + 2>(Sx, P[0] - rA[0], P[0] - rB[0], r2p);
            os_overlap<LA + 1, LB + 2>(Sy, P[1] - rA[1], P[1] - rB[1], r2p);
            os_overlap<LA + 1, LB + 2>(Sz, P[2] - rA[2], P[2] - rB[2], r2p);
            const double sp = PI / p;
            const double pref = sp * sqrt(sp) * pp.K[ip];
#pragma unroll
            for (int ia = 0; ia < NA; ++ia)
#pragma unroll
                for (int jb = 0; jb < NB; ++jb) {
                    const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
                    const int bx = cart_x(LB, jb), by = cart_y(LB, jb), bz = cart_z(LB, jb);
                    const double ox = Sx[ax][bx], oy = Sy[ay][by], oz = Sz[az][bz];
                    const double tx = kin1d<LA + 1, LB + 2>(Sx, ax, bx, b);
                    const double ty = kin1d<LA + 1, LB + 2>(Sy, ay, by, b);
                    const double tz = kin1d<LA + 1, LB + 2>(Sz, az, bz, b);
                    // derivative of the first function along x: 2a S(ax+1) - ax S(ax-1)
                    const double dox = 2.0 * a * Sx[ax + 1][bx] - (ax > 0 ? ax * Sx[ax > 0 ? ax - 1 : 0][bx] : 0.0);
                    const double doy = 2.0 * a * Sy[ay + 1][by] - (ay > 0 ? ay * Sy[ay > 0 ? ay - 1 : 0][by] : 0.0);
                    const double doz = 2.0 * a * Sz[az + 1][bz] - (az > 0 ? az * Sz[az > 0 ? az - 1 : 0][bz] : 0.0);
                    const double dtx = 2.0 * a * kin1d<LA + 1, LB + 2>(Sx, ax + 1, bx, b) -
                                       (ax > 0 ? ax * kin1d<LA + 1, LB + 2>(Sx, ax > 0 ? ax - 1 : 0, bx, b) : 0.0);
                    const double dty = 2.0 * a * kin1d<LA + 1, LB + 2>(Sy, ay + 1, by, b) -
                                       (ay > 0 ? ay * kin1d<LA + 1, LB + 2>(Sy, ay > 0 ? ay - 1 : 0, by, b) : 0.0);
                    const double dtz = 2.0 * a * kin1d<LA + 1, LB + 2>(Sz, az + 1, bz, b) -
                                       (az > 0 ? az * kin1d<LA + 1, LB + 2>(Sz, az > 0 ? az - 1 : 0, bz, b) : 0.0);
                    const double dSx = dox * oy * oz, dSy = ox * doy * oz, dSz = ox * oy * doz;
                    const double dTx = dtx * oy * oz + dox * ty * oz + dox * oy * tz;
                    const double dTy = tx * doy * oz + ox * dty * oz + ox * doy * tz;
                    const double dTz = tx * oy * doz + ox * ty * doz + ox * oy * dtz;
                    const double pw = Pab[ia * NB + jb], ww = Wab[ia * NB + jb];
                    gA[0] += pref * (pw * dTx - ww * dSx);
                    gA[1] += pref * (pw * dTy - ww * dSy);
                    gA[2] += pref * (pw * dTz - ww * dSz);
                }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) gB[d] = -gA[d];  // overlap and kinetic energy: dB = -dA
    }
    int G = 32;  // lanes over nuclei
    while (G / 2 >= bs.natom) G /= 2;
    const double ab[3] = {rA[0] - rB[0], rA[1] - rB[1], rA[2] - rB[2]}, zero[3] = {0.0, 0.0, 0.0};
    for (int c = lane & (G - 1); c < bs.natom; c += G) {
        const double Z = bs.atom_Z[c];
        if (Z == 0.0) continue;
        double gC[3] = {0.0, 0.0, 0.0};
        for (int ip = p0 + lane / G; ip < p0 + np; ip += 32 / G) {
            const double a = pp.a[ip], p = a + pp.b[ip], rs = rsqrt(p + NUC_ZETA), hp = pp.hp[ip];
            const double P[3] = {pp.Px[ip], pp.Py[ip], pp.Pz[ip]};
            const double PA[3] = {P[0] - rA[0], P[1] - rA[1], P[2] - rA[2]}, PB[3] = {P[0] - rB[0], P[1] - rB[1], P[2] - rB[2]};
            const double PC[3] = {P[0] - bs.atom_xyz[3 * c], P[1] - bs.atom_xyz[3 * c + 1], P[2] - bs.atom_xyz[3 * c + 2]};
            double dP[3], da[3], db[3], dc[3], dd[3];
            const double e = md_gradient<LA, LB, 0, 0, double>(p * NUC_ZETA * rs * rs, PC, -Z * NUC_PREF * rs * pp.Kp[ip], PA, PB,
                                                               hp, zero, zero, 0.0, Pab, dP, da, db, dc, dd);
            // P = (a A + b B) / p at fixed A - B; P - A = -(b/p)(A - B), P - B = (a/p)(A - B); exp(-(a b/p) |A-B|^2);
            // translational invariance of each nuclear term: dC = -(dA + dB) = -dP
            const double ap = 2.0 * a * hp, bp = 1.0 - ap, ka = -2.0 * a * bp * e;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double ga = ap * dP[k] + ka * ab[k] - bp * da[k] + ap * db[k];
                gA[k] += ga;
                gB[k] += dP[k] - ga;
                gC[k] -= dP[k];
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(&grad[3 * c + k], gC[k]);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double sa = warp_sum(gA[k]), sb = warp_sum(gB[k]);
        if (lane == 0) {
            atomicAdd(&grad[3 * atA + k], sa);
            atomicAdd(&grad[3 * atB + k], sb);
        }
    }
}

constexpr int PLA[PDG_NPAIRCLASS] = {0, 1, 1, 2, 2, 2};
constexpr int PLB[PDG_NPAIRCLASS] = {0, 0, 1, 0, 1, 2};

template <int C>
void launch_oneint(const pdg_context *ctx, double *S, double *T, double *V, ClassFork &fork) {
    const PairList &pl = ctx->pairs[C];
    if (pl.n == 0) return;
    { oneint_kernel<PLA[C], PLB[C]><<<(pl.n + OPB - 1) / OPB, 32 * OPB, 0, fork.stream(pl.n)>>>(pl, ctx->pp, ctx->dbasis, ctx->nbf, S, T, V); pdg_count_launch(); }
}
template <int C>
void launch_oneint_grad(const pdg_context *ctx, const double *P, const double *W, double *part, int gstride, ClassFork &fork) {
    const PairList &pl = ctx->pairs[C];
    if (pl.n == 0) return;
    { oneint_grad_kernel<PLA[C], PLB[C]><<<(pl.n + OPB - 1) / OPB, 32 * OPB, 0, fork.stream(pl.n)>>>(pl, ctx->pp, ctx->dbasis, ctx->nbf, P, W, part, gstride); pdg_count_launch(); }
}

}  // namespace

int pdg_oneint(pdg_context *ctx, double *d_S, double *d_T, double *d_V) {
    PDG_CHECK(pdg_ensure_pairs(ctx));
    ProfScope prof(ctx, "oneint");
    const size_t nn = (size_t)ctx->nbf * ctx->nbf * sizeof(double);
    PDG_CUDA(cudaMemsetAsync(d_S, 0, nn, ctx->stream));
    PDG_CUDA(cudaMemsetAsync(d_T, 0, nn, ctx->stream));
    PDG_CUDA(cudaMemsetAsync(d_V, 0, nn, ctx->stream));
    ClassFork fork(ctx);
    launch_oneint<0>(ctx, d_S, d_T, d_V, fork);
    launch_oneint<1>(ctx, d_S, d_T, d_V, fork);
    launch_oneint<2>(ctx, d_S, d_T, d_V, fork);
    launch_oneint<3>(ctx, d_S, d_T, d_V, fork);
    launch_oneint<4>(ctx, d_S, d_T, d_V, fork);
    launch_oneint<5>(ctx, d_S, d_T, d_V, fork);
    PDG_CUDA(cudaGetLastError());
    return PDG_OK;
}

int pdg_oneint_grad(pdg_context *ctx, const double *d_P, const double *d_W, double *d_grad) {
    PDG_CHECK(pdg_ensure_pairs(ctx));
    ProfScope prof(ctx, "oneint_grad");
    int gstride = 0;
    double *part = nullptr;
    PDG_CHECK(pdg_grad_part(ctx, &part, &gstride));
    {
        ClassFork fork(ctx);
        launch_oneint_grad<0>(ctx, d_P, d_W, part, gstride, fork);
        launch_oneint_grad<1>(ctx, d_P, d_W, part, gstride, fork);
        launch_oneint_grad<2>(ctx, d_P, d_W, part, gstride, fork);
        launch_oneint_grad<3>(ctx, d_P, d_W, part, gstride, fork);
        launch_oneint_grad<4>(ctx, d_P, d_W, part, gstride, fork);
        launch_oneint_grad<5>(ctx, d_P, d_W, part, gstride, fork);
    }
    PDG_CUDA(cudaGetLastError());
    return pdg_grad_sum(ctx, part, gstride, d_grad);
}
