// Two-electron Coulomb/exchange kernels per angular-momentum class and their launchers.  Included by one
// source file per bra class (eri_jk_<class>.cu), so that the classes compile in parallel, and by eri.cu
// for the Schwarz bounds.
//
// Conventions (all on raw Cartesian integrals; the per-component normalisation n_a is
// folded into D' = N D N on input and F = N F' N on output):
//   for each unique shell quartet (AB|CD), A>=B, C>=D, (AB)>=(CD), degeneracy factor
//   s = 1/2^(#coincidences), full component block V[a][b][c][d]:
//     Jt[a][b] += 2 s sum_cd V D'cd,  Jt[c][d] += 2 s sum_ab V D'ab
//     Kt[a][c] += s sum V D'bd, Kt[a][d] += s sum V D'bc, Kt[b][c] += s sum V D'ad, Kt[b][d] += s sum V D'ac
//   J = Jt + Jt^T, K = Kt + Kt^T, F2 = J - (c_x/2) K, E2 = 1/2 tr(P F2)
// which equals the reference digest, including its 1e-12 storage underflow when
// tei_underflow = 1e-12 (BlockStorage.c:160-181).
#pragma once
#include <atomic>
#include <type_traits>

#include "context.h"
#include "md.cuh"
#include "rys.cuh"
#include "rys2d.cuh"

struct JKArgs {
    PairList bra, ket;
    WorkList work;       // the quartets: per ket bucket, prefix sums over bra pairs and the bra map
    int same;
    PrimPairs pp;
    DeviceBasis bs;
    const double *D;
    double *J, *K;
    int n;
    double underflow;
    const double *dmax;  // optional: max |D'| per shell-pair block (nshell x nshell) for density screening
    int nshell;
    double dcut;         // skip a quartet when Q_AB Q_CD max(relevant dmax) < dcut
    int part;            // 0: every quartet; 1: only bound >= mixed_cut (FP64); 2: only bound < mixed_cut (FP32)
    double mixed_cut;
    int variant;         // host side: lanes-per-bucket table of the launch (-1: by jk_form)
    unsigned long long *count32;  // optional: running count of quartets evaluated in FP32
};

typedef void (*jk_launcher)(const JKArgs &, const QuartetBlock &, bool, bool, bool, cudaStream_t);

// Launchers of a bra class by ket class (eri_jk_<class>.cu).
const jk_launcher *pdg_jk_row0();
const jk_launcher *pdg_jk_row1();
const jk_launcher *pdg_jk_row2();
const jk_launcher *pdg_jk_row3();
const jk_launcher *pdg_jk_row4();
const jk_launcher *pdg_jk_row5();

namespace {

constexpr int PLA[PDG_NPAIRCLASS] = {0, 1, 1, 2, 2, 2};
constexpr int PLB[PDG_NPAIRCLASS] = {0, 0, 1, 0, 1, 2};

// Lanes per quartet for the cooperative form (0: one thread per quartet).
__host__ __device__ constexpr int jk_group(int la, int lb, int lc, int ld) {
    return (la == 2 && lb == 2 && lc == 2 && ld >= 1) ? 32
         : (la == 2 && lb == 2 && lc == 1 && ld == 1) ? 16
         : (la == 2 && lb == 1 && lc == 2 && ld == 1) ? 16
         : (la == 2 && lb == 2 && lc == 2 && ld == 0) ? 16
         : (la == 2 && lb == 1 && lc == 1 && ld == 1) ? 8
         : (la == 2 && lb == 2 && lc == 1 && ld == 0) ? 8
         : (la == 2 && lb == 1 && lc == 2 && ld == 0) ? 8
         : 0;
}

// The classes of small component blocks (up to 36) split their primitive quartets over lanes, more lanes
// for the ket buckets with more primitive pairs; the wider blocks only in short lists (kWideLanes).
__host__ __device__ constexpr bool jk_split(int la, int lb, int lc, int ld) {
    return ncart(la) * ncart(lb) * ncart(lc) * ncart(ld) <= 36;
}
// Lanes per quartet by ket bucket for the small-block classes in lists below kWarpItems: five tables, taken
// by the length of the list (jk_form) from the class pair's first one on (pair classes ss, ps, pp, ds, dp,
// dd), or as pdg_autotune_eri chose.  The first ones are what it chose on a 14-heavy-atom organic molecule in
// B3LYP/6-31G* (Cartesian) when its lists took tables: table 3 (2-16 lanes) for (ss|ss), table 0 for (dp|ss)
// and (dd|ss), table 1 for the rest.
constexpr int kNLanesV = 5;
constexpr int kSplitLanesV[kNLanesV][PDG_NBUCKET] = {
    {1, 1, 1, 2, 2}, {1, 1, 2, 4, 4}, {1, 2, 4, 8, 8}, {2, 4, 8, 16, 16}, {4, 8, 16, 32, 32}};
constexpr int kDefaultLanesV[PDG_NPAIRCLASS][PDG_NPAIRCLASS] = {
    {3, 1, 1, 1, 1, 1}, {1, 1, 1, 1, 1, 1}, {1, 1, 1, 1, 1, 1},
    {1, 1, 1, 1, 1, 1}, {0, 1, 1, 1, 1, 1}, {0, 1, 1, 1, 1, 1}};
// Lists of at least this many (bra, ket group) items take the warp-per-bra form; one lane then walks all
// primitives of a quartet, so a shorter list leaves the chip waiting for its longest quartets and keeps
// several lanes per quartet.  J+K builds with the line at 2368, 8192, 32768 items and with no warp form at
// all: 4 waters 349, 231, 233, 233 us; 6 waters 626, 631, 493, 490; 8 waters 808, 854, 936, 936; 16 waters 4096,
// 4144, 4375, 5338; 42 atoms 11.13, 11.12, 11.47, 14.41 ms (the mixed mode alike).
constexpr long long kWarpItems = 8192;
// A list of few quartets takes the tables of more lanes while its threads stay below kLaneThreads, one to
// two times those that fit the chip's 148 SMs at the kernels' registers: the launch then lasts as long as its
// longest quartet, and one lane takes 0.2 ms for the 81 primitive quartets of a (pp|pp) one.  Lanes beyond that
// only repeat the quartets' preambles.  The same for the classes of wide blocks, from one lane per
// quartet and at half the threads (255 registers).  J+K builds with no more lanes than the first table's, with
// this limit and with eight times it: one water 315, 162, 159 us; 4 waters 341, 234, 242; 8 waters 917, 860, 1091;
// 16 heavy and hydrogen atoms (5 heavy) 544, 525, 630.
constexpr long long kLaneThreads = 148 * 1024;
constexpr int kNWide = 4;
constexpr int kWideLanes[kNWide][PDG_NBUCKET] = {{1, 1, 1, 1, 1}, {1, 2, 2, 2, 2}, {2, 4, 4, 4, 4}, {4, 8, 8, 8, 8}};

}  // namespace

// The table that pdg_autotune_eri chose for each (bra class, ket class), for every context of the process (-1:
// none, by the length of the list).
extern std::atomic<int> pdg_jk_variant[PDG_NPAIRCLASS][PDG_NPAIRCLASS];

namespace {

// The form of a list of a class pair without cooperative kernel: kWarpForm, or the table of lanes (of
// kSplitLanesV or kWideLanes).
constexpr int kWarpForm = 8;
inline int jk_form(const QuartetBlock &b) {
    if (pdg_warp_items(b) >= kWarpItems) return kWarpForm;
    int v = 0;
    if (jk_split(PLA[b.cb], PLB[b.cb], PLA[b.ck], PLB[b.ck])) {
        v = pdg_jk_variant[b.cb][b.ck].load(std::memory_order_relaxed);
        if (v >= 0) return v;
        v = kDefaultLanesV[b.cb][b.ck];
        while (v + 1 < kNLanesV && pdg_work_threads(b, kSplitLanesV[v + 1]) <= kLaneThreads) ++v;
    } else {
        while (v + 1 < kNWide && pdg_work_threads(b, kWideLanes[v + 1]) <= kLaneThreads / 2) ++v;
    }
    return v;
}

constexpr double TWO_PI_POW_2P5 = 34.986836655249725;  // 2 pi^(5/2)

__host__ __device__ constexpr double comp_norm(int l, int i) {
    // sqrt((2l-1)!! / ((2x-1)!! (2y-1)!! (2z-1)!!)) for l <= 2: only xy, xz, yz differ from 1.
    return (l == 2 && (i == 1 || i == 3 || i == 4)) ? 1.7320508075688772 : 1.0;
}

struct QuartetGeom {
    double A[3], B[3], C[3], D[3];
};

// One primitive quartet (bra primitive pair B, ket primitive pair K) added to the raw Cartesian
// block V[(a*NB+b)*NC*ND + c*ND + d].  T is the arithmetic type of the recursions and the
// accumulation (float for the quartets of the mixed-precision mode); the Boys argument, the Rys
// rule and the prefactors stay in double.
template <int LA, int LB, int LC, int LD, typename T = double>
__device__ __forceinline__ void eri_prim(const PairRec &B, const PairRec &K, const QuartetGeom &g,
                                         T (&V)[ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD)]) {
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int LAB = LA + LB, LCD = LC + LD, NR = (LAB + LCD) / 2 + 1;
    const double p = B.p, Px = B.Px, Py = B.Py, Pz = B.Pz;
    const double q = K.p, Qx = K.Px, Qy = K.Py, Qz = K.Pz;
    const double rs = rsqrt(p + q), rppq = rs * rs;
    const double PQx = Px - Qx, PQy = Py - Qy, PQz = Pz - Qz;
    const double x = p * q * rppq * (PQx * PQx + PQy * PQy + PQz * PQz);
    const double pref = TWO_PI_POW_2P5 * rs * B.Kp * K.Kp;
    if constexpr (md_class(LA, LB, LC, LD) && std::is_same<T, double>::value) {
        const double PQ[3] = {PQx, PQy, PQz};
        const double PA[3] = {Px - g.A[0], Py - g.A[1], Pz - g.A[2]}, PB[3] = {Px - g.B[0], Py - g.B[1], Pz - g.B[2]};
        const double QC[3] = {Qx - g.C[0], Qy - g.C[1], Qz - g.C[2]}, QD[3] = {Qx - g.D[0], Qy - g.D[1], Qz - g.D[2]};
        md_energy<LA, LB, LC, LD, double>(p * q * rppq, PQ, pref, PA, PB, B.hp, QC, QD, K.hp, V);
        return;
    }
    double u[NR], w[NR];
    rys_roots<NR>(x, u, w);
    const double PAx = Px - g.A[0], PAy = Py - g.A[1], PAz = Pz - g.A[2];
    const double QCx = Qx - g.C[0], QCy = Qy - g.C[1], QCz = Qz - g.C[2];
    const T ABx = T(g.A[0] - g.B[0]), ABy = T(g.A[1] - g.B[1]), ABz = T(g.A[2] - g.B[2]);
    const T CDx = T(g.C[0] - g.D[0]), CDy = T(g.C[1] - g.D[1]), CDz = T(g.C[2] - g.D[2]);
    const double r2p = B.hp, r2q = K.hp;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const double ur = u[r] * rppq;
        const T b00 = T(0.5 * ur);
        const T b10 = T(r2p * (1.0 - q * ur));
        const T b01 = T(r2q * (1.0 - p * ur));
        const double fq = q * ur, fp = p * ur;
        T Gx[LAB + 1][LCD + 1], Gy[LAB + 1][LCD + 1], Gz[LAB + 1][LCD + 1];
        rys_vrr<LAB, LCD, T>(Gx, T(1), T(PAx - fq * PQx), T(QCx + fp * PQx), b10, b01, b00);
        rys_vrr<LAB, LCD, T>(Gy, T(1), T(PAy - fq * PQy), T(QCy + fp * PQy), b10, b01, b00);
        rys_vrr<LAB, LCD, T>(Gz, T(w[r] * pref), T(PAz - fq * PQz), T(QCz + fp * PQz), b10, b01, b00);
        T Ix[LA + 1][LB + 1][LC + 1][LD + 1], Iy[LA + 1][LB + 1][LC + 1][LD + 1], Iz[LA + 1][LB + 1][LC + 1][LD + 1];
        rys_hrr<LA, LB, LC, LD, T>(Gx, ABx, CDx, Ix);
        rys_hrr<LA, LB, LC, LD, T>(Gy, ABy, CDy, Iy);
        rys_hrr<LA, LB, LC, LD, T>(Gz, ABz, CDz, Iz);
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
            for (int jb = 0; jb < NB; ++jb)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc)
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const T vx = Ix[cart_x(LA, ia)][cart_x(LB, jb)][cart_x(LC, kc)][cart_x(LD, ld)];
                        const T vy = Iy[cart_y(LA, ia)][cart_y(LB, jb)][cart_y(LC, kc)][cart_y(LD, ld)];
                        const T vz = Iz[cart_z(LA, ia)][cart_z(LB, jb)][cart_z(LC, kc)][cart_z(LD, ld)];
                        V[((ia * NB + jb) * NC + kc) * ND + ld] += vx * vy * vz;
                    }
    }
}

// Quartet geometry for the FP32 quartets: the centre differences, taken in double and rounded once.
struct QuartetGeom32 {
    float ABx, ABy, ABz, CDx, CDy, CDz, ACx, ACy, ACz;
};
__device__ __forceinline__ QuartetGeom32 geom32(const QuartetGeom &g) {
    return QuartetGeom32{(float)(g.A[0] - g.B[0]), (float)(g.A[1] - g.B[1]), (float)(g.A[2] - g.B[2]),
                         (float)(g.C[0] - g.D[0]), (float)(g.C[1] - g.D[1]), (float)(g.C[2] - g.D[2]),
                         (float)(g.A[0] - g.C[0]), (float)(g.A[1] - g.C[1]), (float)(g.A[2] - g.C[2])};
}

// eri_prim entirely in single precision, for the quartets of the mixed mode whose bound is below the
// mixed cut: Boys argument, Rys rule (rys_roots_f), prefactor, recursions and accumulation.  With
// P - A and Q - C from the records, P - Q = (P - A) - (Q - C) + (A - C).
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void eri_prim32(const PairRec32 &B, const PairRec32 &K, const QuartetGeom32 &g,
                                           float (&V)[ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD)]) {
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int LAB = LA + LB, LCD = LC + LD, NR = (LAB + LCD) / 2 + 1;
    const float p = B.p, q = K.p;
    const float rs = rsqrtf(p + q), rppq = rs * rs;
    const float PQx = B.PAx - K.PAx + g.ACx, PQy = B.PAy - K.PAy + g.ACy, PQz = B.PAz - K.PAz + g.ACz;
    const float x = p * q * rppq * (PQx * PQx + PQy * PQy + PQz * PQz);
    const float pref = (float)TWO_PI_POW_2P5 * rs * B.Kp * K.Kp;
    if constexpr (md_class(LA, LB, LC, LD)) {
        const float PQ[3] = {PQx, PQy, PQz}, PA[3] = {B.PAx, B.PAy, B.PAz}, QC[3] = {K.PAx, K.PAy, K.PAz};
        const float PB[3] = {B.PAx + g.ABx, B.PAy + g.ABy, B.PAz + g.ABz}, QD[3] = {K.PAx + g.CDx, K.PAy + g.CDy, K.PAz + g.CDz};
        md_energy<LA, LB, LC, LD, float>(p * q * rppq, PQ, pref, PA, PB, B.hp, QC, QD, K.hp, V);
        return;
    }
    float u[NR], w[NR];
    rys_roots_f<NR>(x, u, w);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const float ur = u[r] * rppq;
        const float b00 = 0.5f * ur, b10 = B.hp * (1.0f - q * ur), b01 = K.hp * (1.0f - p * ur);
        const float fq = q * ur, fp = p * ur;
        float Gx[LAB + 1][LCD + 1], Gy[LAB + 1][LCD + 1], Gz[LAB + 1][LCD + 1];
        rys_vrr<LAB, LCD, float>(Gx, 1.0f, B.PAx - fq * PQx, K.PAx + fp * PQx, b10, b01, b00);
        rys_vrr<LAB, LCD, float>(Gy, 1.0f, B.PAy - fq * PQy, K.PAy + fp * PQy, b10, b01, b00);
        rys_vrr<LAB, LCD, float>(Gz, w[r] * pref, B.PAz - fq * PQz, K.PAz + fp * PQz, b10, b01, b00);
        float Ix[LA + 1][LB + 1][LC + 1][LD + 1], Iy[LA + 1][LB + 1][LC + 1][LD + 1], Iz[LA + 1][LB + 1][LC + 1][LD + 1];
        rys_hrr<LA, LB, LC, LD, float>(Gx, g.ABx, g.CDx, Ix);
        rys_hrr<LA, LB, LC, LD, float>(Gy, g.ABy, g.CDy, Iy);
        rys_hrr<LA, LB, LC, LD, float>(Gz, g.ABz, g.CDz, Iz);
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
            for (int jb = 0; jb < NB; ++jb)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc)
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const float vx = Ix[cart_x(LA, ia)][cart_x(LB, jb)][cart_x(LC, kc)][cart_x(LD, ld)];
                        const float vy = Iy[cart_y(LA, ia)][cart_y(LB, jb)][cart_y(LC, kc)][cart_y(LD, ld)];
                        const float vz = Iz[cart_z(LA, ia)][cart_z(LB, jb)][cart_z(LC, kc)][cart_z(LD, ld)];
                        V[((ia * NB + jb) * NC + kc) * ND + ld] += vx * vy * vz;
                    }
    }
}

__device__ __forceinline__ void load_xyz(const DeviceBasis &bs, int sh, double *r) {
    const int at = bs.sh_atom[sh];
    r[0] = bs.atom_xyz[3 * at];
    r[1] = bs.atom_xyz[3 * at + 1];
    r[2] = bs.atom_xyz[3 * at + 2];
}

// Adds the quartets of the calling lanes that lead a quartet (leader) to args.count32, one atomic
// per warp.
__device__ __forceinline__ void count_fp32(const JKArgs &args, bool leader) {
    if (!args.count32 || args.part != 2) return;
    const unsigned am = __activemask();
    const unsigned bm = __ballot_sync(am, leader);
    if (leader && (int)(threadIdx.x & 31) == __ffs(bm) - 1) atomicAdd(args.count32, (unsigned long long)__popc(bm));
}

// Density screening and the precision partition of the mixed mode.  The Coulomb and exchange
// parts are screened separately: a quartet changes J by at most Q_AB Q_CD max(|D_AB|, |D_CD|) and
// K by at most Q_AB Q_CD max(|D_AC|, |D_AD|, |D_BC|, |D_BD|); each part is digested only when its
// bound reaches dcut, and the quartet is skipped when neither does.  The mixed mode partitions on
// the larger of the two bounds.
struct JKScreen {
    bool any, j, k;
};
template <bool DOJ, bool DOK>
__device__ __forceinline__ JKScreen jk_screen(const JKArgs &args, int ib, int ik, int A, int B, int C, int D) {
    if (!args.dmax) return {true, DOJ, DOK};
    const int ns = args.nshell;
    const double q = args.bra.Q[ib] * args.ket.Q[ik];
    const double bj = DOJ ? q * fmax(args.dmax[A * ns + B], args.dmax[C * ns + D]) : 0.0;
    const double bk = DOK ? q * fmax(fmax(args.dmax[B * ns + D], args.dmax[B * ns + C]),
                                     fmax(args.dmax[A * ns + D], args.dmax[A * ns + C])) : 0.0;
    JKScreen r{false, DOJ && bj >= args.dcut, DOK && bk >= args.dcut};
    r.any = r.j || r.k;
    const double bound = fmax(bj, bk);
    if (args.part == 1) r.any = r.any && bound >= args.mixed_cut;
    if (args.part == 2) r.any = r.any && bound < args.mixed_cut;
    return r;
}

// One shell quartet per P lanes (the bucket's lane count, 1 to 32): the lanes split
// the primitive quartets and add their blocks with shuffles; the first lanes digest, one the J part
// and up to two the K parts (rows of a, rows of b), as independent streams of loads and atomics that
// the warp scheduler interleaves.  Splitting keeps more primitive loads in flight for the contracted
// s/p classes (up to 6 x 6 primitive pairs per shell pair), whose one-lane loops are bound by load
// latency; the ket buckets give the quartets of a warp the same primitive count.
template <int LA, int LB, int LC, int LD, bool DOJ, bool DOK, typename T>
__global__ void __launch_bounds__(128) eri_jk_kernel(JKArgs args) {
    const WorkSub ws = pick_sub(args.work);
    const int P = ws.lanes;
    const long long t = ((long long)blockIdx.x - ws.cta0) * blockDim.x / P + (long long)(threadIdx.x / P);
    const int lane = (int)(threadIdx.x & (P - 1));
    const int ib = bra_of(ws.offs, ws.cbra, min(t, ws.total - 1));
    if (t >= ws.total) return;
    const int ik = ws.k0 + (int)(t - ws.offs[ib]);
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    const int A = args.bra.shA[ib], B = args.bra.shB[ib], C = args.ket.shA[ik], D = args.ket.shB[ik];
    // density screening: the quartet changes J (K) by at most Q_AB Q_CD times the largest
    // density element it is contracted with
    const JKScreen scr = jk_screen<DOJ, DOK>(args, ib, ik, A, B, C, D);
    if (!scr.any) return;
    count_fp32(args, lane == 0);
    QuartetGeom g;
    load_xyz(args.bs, A, g.A);
    load_xyz(args.bs, B, g.B);
    load_xyz(args.bs, C, g.C);
    load_xyz(args.bs, D, g.D);
    T V[NA * NB * NC * ND];
#pragma unroll
    for (int i = 0; i < NA * NB * NC * ND; ++i) V[i] = T(0);
    const int pb0 = args.bra.poff[ib], pk0 = args.ket.poff[ik], npk = args.ket.np[ik];
    const int nprim = args.bra.np[ib] * npk;
    // primitive quartet idx = jb npk + jk, stepped by P without a division per step
    int jb = lane / npk, jk = lane - jb * npk;
    if constexpr (std::is_same<T, float>::value) {
        const QuartetGeom32 g32 = geom32(g);
        for (int idx = lane; idx < nprim; idx += P, jk += P) {
            while (jk >= npk) { jk -= npk; ++jb; }
            const PairRec32 Bp = load_rec32(args.pp.rec32, pb0 + jb), Kp = load_rec32(args.pp.rec32, pk0 + jk);
            if (Bp.arg + Kp.arg > (float)PDG_PRIMITIVE_CUT) continue;
            eri_prim32<LA, LB, LC, LD>(Bp, Kp, g32, V);
        }
    } else {
        for (int idx = lane; idx < nprim; idx += P, jk += P) {
            while (jk >= npk) { jk -= npk; ++jb; }
            const int xb = pb0 + jb, xk = pk0 + jk;
            if (load_arg(args.pp.rec, xb) + load_arg(args.pp.rec, xk) > PDG_PRIMITIVE_CUT) continue;
            eri_prim<LA, LB, LC, LD, T>(load_rec(args.pp.rec, xb), load_rec(args.pp.rec, xk), g, V);
        }
    }
    const unsigned mask = lane_group_mask(P);
    for (int o = P >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int i = 0; i < NA * NB * NC * ND; ++i) V[i] += __shfl_xor_sync(mask, V[i], o);
    }
    // every lane of the group now holds the contracted block; up to three of them share the
    // digest (J; K rows of a; K rows of b)
    if (lane >= (P < 3 ? P : 3)) return;
    const int roles = P < 3 ? P : 3;
    const bool do_j = lane == 0;
    const bool do_ka = roles == 3 ? lane == 1 : lane == 0;
    const bool do_kb = lane == roles - 1;
    double s = 1.0;
    if (A == B) s *= 0.5;
    if (C == D) s *= 0.5;
    if (args.same && ib == ik) s *= 0.5;
    const double uf = args.underflow;
    if (uf > 0.0) {
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
            for (int jb = 0; jb < NB; ++jb)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc)
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const int f = ((ia * NB + jb) * NC + kc) * ND + ld;
                        const double nn = comp_norm(LA, ia) * comp_norm(LB, jb) * comp_norm(LC, kc) * comp_norm(LD, ld);
                        if (fabs((double)V[f] * nn) <= uf) V[f] = T(0);
                    }
    }
    const int n = args.n;
    const int oa = args.bs.sh_bf[A], ob = args.bs.sh_bf[B], oc = args.bs.sh_bf[C], od = args.bs.sh_bf[D];
    const double *__restrict__ Dm = args.D;
    if (DOJ && scr.j && do_j) {
        const double s2 = 2.0 * s;
        double dcd[NC * ND];
#pragma unroll
        for (int kc = 0; kc < NC; ++kc)
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) dcd[kc * ND + ld] = Dm[(oc + kc) * n + od + ld];
        double jcd[NC * ND];
#pragma unroll
        for (int i = 0; i < NC * ND; ++i) jcd[i] = 0.0;
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
            for (int jb = 0; jb < NB; ++jb) {
                const double dab = Dm[(oa + ia) * n + ob + jb];
                double jab = 0.0;
#pragma unroll
                for (int kl = 0; kl < NC * ND; ++kl) {
                    const double v = V[(ia * NB + jb) * NC * ND + kl];
                    jab += v * dcd[kl];
                    jcd[kl] += v * dab;
                }
                atomicAdd(&args.J[(oa + ia) * n + ob + jb], s2 * jab);
            }
#pragma unroll
        for (int kc = 0; kc < NC; ++kc)
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) atomicAdd(&args.J[(oc + kc) * n + od + ld], s2 * jcd[kc * ND + ld]);
    }
    if (DOK && scr.k && do_ka) {
        // Kt[a][c] += s V Dbd ; Kt[a][d] += s V Dbc
#pragma unroll
        for (int ia = 0; ia < NA; ++ia) {
            double kac[NC], kad[ND];
#pragma unroll
            for (int i = 0; i < NC; ++i) kac[i] = 0.0;
#pragma unroll
            for (int i = 0; i < ND; ++i) kad[i] = 0.0;
#pragma unroll
            for (int jb = 0; jb < NB; ++jb)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc) {
                    const double dbc = Dm[(ob + jb) * n + oc + kc];
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const double v = V[((ia * NB + jb) * NC + kc) * ND + ld];
                        kac[kc] += v * Dm[(ob + jb) * n + od + ld];
                        kad[ld] += v * dbc;
                    }
                }
#pragma unroll
            for (int kc = 0; kc < NC; ++kc) atomicAdd(&args.K[(oa + ia) * n + oc + kc], s * kac[kc]);
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) atomicAdd(&args.K[(oa + ia) * n + od + ld], s * kad[ld]);
        }
    }
    if (DOK && scr.k && do_kb) {
        // Kt[b][c] += s V Dad ; Kt[b][d] += s V Dac
#pragma unroll
        for (int jb = 0; jb < NB; ++jb) {
            double kbc[NC], kbd[ND];
#pragma unroll
            for (int i = 0; i < NC; ++i) kbc[i] = 0.0;
#pragma unroll
            for (int i = 0; i < ND; ++i) kbd[i] = 0.0;
#pragma unroll
            for (int ia = 0; ia < NA; ++ia)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc) {
                    const double dac = Dm[(oa + ia) * n + oc + kc];
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const double v = V[((ia * NB + jb) * NC + kc) * ND + ld];
                        kbc[kc] += v * Dm[(oa + ia) * n + od + ld];
                        kbd[ld] += v * dac;
                    }
                }
#pragma unroll
            for (int kc = 0; kc < NC; ++kc) atomicAdd(&args.K[(ob + jb) * n + oc + kc], s * kbc[kc]);
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) atomicAdd(&args.K[(ob + jb) * n + od + ld], s * kbd[ld]);
        }
    }
}

// Sum over the warp; every lane takes part.
__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp per (bra pair, group of 32 kets): a lane holds one quartet.  The bra is the same for all
// lanes, so its records come as broadcast loads and its J elements leave as one atomic per warp; the
// kets' records come from the group layout in whole lines, once per ket primitive (outer loop) for all
// bra primitives.  The form with lanes split over the primitives of a quartet reads both records as
// gathers, repeats the quartet's preamble in every lane and adds J_ab once per lane to one address; the
// L1 data pipe was 81-92% busy there, here 48-64% with the FP64 pipe at 31-44%.  J+K build of a 42-atom
// molecule (266 functions, B3LYP) 15.7 -> 13.4 ms, of a 63-atom one in the mixed mode 73.1 -> 59.6 ms.
template <int LA, int LB, int LC, int LD, bool DOJ, bool DOK, typename T>
__global__ void __launch_bounds__(128) eri_jk_warp_kernel(JKArgs args) {
    const WorkSub ws = pick_sub(args.work);
    const long long w = ((long long)blockIdx.x - ws.cta0) * 4 + (threadIdx.x >> 5);
    if (w >= ws.wtotal) return;
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    const int lane = threadIdx.x & 31;
    const int ib = bra_of(ws.woffs, ws.wbra, w);
    const int grp = (int)(w - ws.woffs[ib]);
    const int cnt = (int)(ws.offs[ib + 1] - ws.offs[ib]), slot = grp * 32 + lane;
    bool act = slot < cnt;
    const int ik = ws.k0 + min(slot, cnt - 1);
    const int A = args.bra.shA[ib], B = args.bra.shB[ib], C = args.ket.shA[ik], D = args.ket.shB[ik];
    const JKScreen scr = jk_screen<DOJ, DOK>(args, ib, ik, A, B, C, D);
    act = act && scr.any;
    const unsigned live = __ballot_sync(0xffffffffu, act);
    if (live == 0) return;
    if (args.count32 && args.part == 2 && lane == 0) atomicAdd(args.count32, (unsigned long long)__popc(live));
    T V[NA * NB * NC * ND];
#pragma unroll
    for (int i = 0; i < NA * NB * NC * ND; ++i) V[i] = T(0);
    if (act) {
        QuartetGeom g;
        load_xyz(args.bs, A, g.A);
        load_xyz(args.bs, B, g.B);
        load_xyz(args.bs, C, g.C);
        load_xyz(args.bs, D, g.D);
        const int pb0 = args.bra.poff[ib], pb1 = pb0 + args.bra.np[ib], npk = args.ket.np[ik];
        const size_t k0 = args.ket.goff[ws.g0 + grp];
        for (int j = 0; j < npk; ++j) {
            if constexpr (std::is_same<T, float>::value) {
                const QuartetGeom32 g32 = geom32(g);
                const PairRec32 Kp = load_grec32(args.ket.grec32, k0 + j);
                for (int xb = pb0; xb < pb1; ++xb) {
                    const PairRec32 Bp = load_rec32(args.pp.rec32, xb);
                    if (Bp.arg + Kp.arg > (float)PDG_PRIMITIVE_CUT) continue;
                    eri_prim32<LA, LB, LC, LD>(Bp, Kp, g32, V);
                }
            } else {
                const double argk = load_grec_arg_a(args.ket.grec, k0 + j).x;
                const PairRec Kp = load_grec(args.ket.grec, k0 + j);
                for (int xb = pb0; xb < pb1; ++xb) {
                    if (load_arg(args.pp.rec, xb) + argk > PDG_PRIMITIVE_CUT) continue;
                    eri_prim<LA, LB, LC, LD, T>(load_rec(args.pp.rec, xb), Kp, g, V);
                }
            }
        }
    }
    __syncwarp();
    const double uf = args.underflow;
    if (uf > 0.0) {
#pragma unroll
        for (int f = 0; f < NA * NB * NC * ND; ++f) {
            const double nn = comp_norm(LA, f / (NB * NC * ND)) * comp_norm(LB, f / (NC * ND) % NB) *
                              comp_norm(LC, f / ND % NC) * comp_norm(LD, f % ND);
            if (fabs((double)V[f] * nn) <= uf) V[f] = T(0);
        }
    }
    double s = 1.0;
    if (A == B) s *= 0.5;
    if (C == D) s *= 0.5;
    if (args.same && ib == ik) s *= 0.5;
    const int n = args.n;
    const int oa = args.bs.sh_bf[A], ob = args.bs.sh_bf[B], oc = args.bs.sh_bf[C], od = args.bs.sh_bf[D];
    const double *__restrict__ Dm = args.D;
    const bool doj = DOJ && act && scr.j;
    if (DOJ && __any_sync(0xffffffffu, doj)) {
        const double s2 = doj ? 2.0 * s : 0.0;
        double dcd[NC * ND], jcd[NC * ND];
#pragma unroll
        for (int i = 0; i < NC * ND; ++i) {
            dcd[i] = Dm[(oc + i / ND) * n + od + i % ND];
            jcd[i] = 0.0;
        }
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
            for (int jb = 0; jb < NB; ++jb) {
                const double dab = Dm[(oa + ia) * n + ob + jb];
                double jab = 0.0;
#pragma unroll
                for (int kl = 0; kl < NC * ND; ++kl) {
                    const double v = V[(ia * NB + jb) * NC * ND + kl];
                    jab += v * dcd[kl];
                    jcd[kl] += v * dab;
                }
                jab = warp_total(s2 * jab);
                if (lane == 0) atomicAdd(&args.J[(oa + ia) * n + ob + jb], jab);
            }
        if (doj) {
#pragma unroll
            for (int i = 0; i < NC * ND; ++i) atomicAdd(&args.J[(oc + i / ND) * n + od + i % ND], s2 * jcd[i]);
        }
    }
    if (DOK && act && scr.k) {
        // Kt[a][c] += s V Dbd ; Kt[a][d] += s V Dbc
#pragma unroll
        for (int ia = 0; ia < NA; ++ia) {
            double kac[NC], kad[ND];
#pragma unroll
            for (int i = 0; i < NC; ++i) kac[i] = 0.0;
#pragma unroll
            for (int i = 0; i < ND; ++i) kad[i] = 0.0;
#pragma unroll
            for (int jb = 0; jb < NB; ++jb)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc) {
                    const double dbc = Dm[(ob + jb) * n + oc + kc];
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const double v = V[((ia * NB + jb) * NC + kc) * ND + ld];
                        kac[kc] += v * Dm[(ob + jb) * n + od + ld];
                        kad[ld] += v * dbc;
                    }
                }
#pragma unroll
            for (int kc = 0; kc < NC; ++kc) atomicAdd(&args.K[(oa + ia) * n + oc + kc], s * kac[kc]);
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) atomicAdd(&args.K[(oa + ia) * n + od + ld], s * kad[ld]);
        }
        // Kt[b][c] += s V Dad ; Kt[b][d] += s V Dac
#pragma unroll
        for (int jb = 0; jb < NB; ++jb) {
            double kbc[NC], kbd[ND];
#pragma unroll
            for (int i = 0; i < NC; ++i) kbc[i] = 0.0;
#pragma unroll
            for (int i = 0; i < ND; ++i) kbd[i] = 0.0;
#pragma unroll
            for (int ia = 0; ia < NA; ++ia)
#pragma unroll
                for (int kc = 0; kc < NC; ++kc) {
                    const double dac = Dm[(oa + ia) * n + oc + kc];
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld) {
                        const double v = V[((ia * NB + jb) * NC + kc) * ND + ld];
                        kbc[kc] += v * Dm[(oa + ia) * n + od + ld];
                        kbd[ld] += v * dac;
                    }
                }
#pragma unroll
            for (int kc = 0; kc < NC; ++kc) atomicAdd(&args.K[(ob + jb) * n + oc + kc], s * kbc[kc]);
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) atomicAdd(&args.K[(ob + jb) * n + od + ld], s * kbd[ld]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Cooperative form for the d-shell classes whose component block (up to 6^4 = 1296 values) does
// not fit one thread's registers: G lanes of a warp share one shell quartet.
//  - per primitive quartet, lanes take the 3 x n_R (root, direction) tasks: one Rys node each
//    (rys_root_single), the 2D recursion and the closed-form transfers
//    I(a,b,c,d) = sum_k sum_m C(b,k) (A-B)^(b-k) C(d,m) (C-D)^(d-m) G(a+k, c+m), written to
//    shared memory;
//  - each lane owns whole bra rows (a,b) of the block (all c,d) and accumulates them over roots
//    and primitives in registers; rows left over after the full rounds are split by c.  Lanes
//    of a row share the (a_x,b_x) slice of the 2D integrals, so a warp load touches at most 9
//    distinct words and is served in one wavefront;
//  - the contracted block is written to shared memory (after the storage underflow) and the
//    J/K digest is spread over the lanes with the needed density blocks staged beside it.
// ---------------------------------------------------------------------------------------------
__host__ __device__ constexpr int binom_small(int n, int k) { return (k == 0 || k == n) ? 1 : (n == 2 ? 2 : n); }

template <int LA, int LB, int LC, int LD, typename T = double>
__device__ __forceinline__ void hrr_store(const T (&Gm)[LA + LB + 1][LC + LD + 1], T AB, T CD, T *__restrict__ out) {
    constexpr int LCD = LC + LD;
    T abp[LB + 1], cdp[LD + 1];
    abp[0] = T(1);
#pragma unroll
    for (int k = 1; k <= LB; ++k) abp[k] = abp[k - 1] * AB;
    cdp[0] = T(1);
#pragma unroll
    for (int k = 1; k <= LD; ++k) cdp[k] = cdp[k - 1] * CD;
#pragma unroll
    for (int a = 0; a <= LA; ++a)
#pragma unroll
        for (int b = 0; b <= LB; ++b) {
            T row[LCD + 1];
#pragma unroll
            for (int f = 0; f <= LCD; ++f) {
                T s = Gm[a + b][f];
#pragma unroll
                for (int k = 0; k < b; ++k) s += T(binom_small(b, k)) * abp[b - k] * Gm[a + k][f];
                row[f] = s;
            }
#pragma unroll
            for (int c = 0; c <= LC; ++c)
#pragma unroll
                for (int d = 0; d <= LD; ++d) {
                    T s = row[c + d];
#pragma unroll
                    for (int m = 0; m < d; ++m) s += T(binom_small(d, m)) * cdp[d - m] * row[c + m];
                    out[((a * (LB + 1) + b) * (LC + 1) + c) * (LD + 1) + d] = s;
                }
        }
}

template <int LA, int LB, int LC, int LD, int G>
struct GroupShape {
    static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    static constexpr int NCD = NC * ND;
    static constexpr int NR = (LA + LB + LC + LD) / 2 + 1;
    static constexpr int NI = (LA + 1) * (LB + 1) * (LC + 1) * (LD + 1);
    static constexpr int NCOMP = NA * NB * NC * ND;
    static constexpr int R = NA * NB;            // bra rows
    static constexpr int FR = R / G;             // full rounds of rows per lane
    static constexpr int LR = R - FR * G;        // rows left over, split by c into units
    static constexpr int NUNIT = LR * NC;
    static constexpr int NU = (NUNIT + G - 1) / G;
    static constexpr int NIP = NI | 1;           // odd strides keep the lanes' rows in distinct banks
    static constexpr int NCDP = NCD | 1;
    static constexpr int NDBLK = NA * NB + NC * ND + NA * NC + NA * ND + NB * NC + NB * ND;
    static constexpr int WORK = (3 * NR * NIP > R * NCDP) ? 3 * NR * NIP : R * NCDP;
    static constexpr int SMEM = WORK + NDBLK;    // doubles per group
    static constexpr int GPB = 128 / G;          // groups per 128-thread block
};

template <int LA, int LB, int LC, int LD, int G, bool DOJ, bool DOK, typename T = double>
__global__ void __launch_bounds__(128) eri_jk_group_kernel(JKArgs args) {
    using S = GroupShape<LA, LB, LC, LD, G>;
    constexpr int NA = S::NA, NB = S::NB, NC = S::NC, ND = S::ND, NCD = S::NCD, NR = S::NR, NI = S::NIP;
    constexpr int NCDP = S::NCDP;  // row stride of the contracted block in shared memory
    constexpr int LAB = LA + LB, LCD = LC + LD;
    extern __shared__ double gsm[];
    const int gq = threadIdx.x / G, lane = threadIdx.x % G;
    double *__restrict__ sm = gsm + gq * S::SMEM;
    double *__restrict__ sD = sm + S::WORK;
    T *__restrict__ sI = reinterpret_cast<T *>(sm);  // 2D integrals during the primitive loop
    const unsigned mask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) / G * G));
    const WorkSub ws = pick_sub(args.work);
    const long long t = ((long long)blockIdx.x - ws.cta0) * S::GPB + gq;
    const int ib = bra_of(ws.offs, ws.cbra, min(t, ws.total - 1));
    if (t >= ws.total) return;
    const int ik = ws.k0 + (int)(t - ws.offs[ib]);
    const int A = args.bra.shA[ib], B = args.bra.shB[ib], C = args.ket.shA[ik], D = args.ket.shB[ik];
    const JKScreen scr = jk_screen<DOJ, DOK>(args, ib, ik, A, B, C, D);
    if (!scr.any) return;
    count_fp32(args, lane == 0);
    QuartetGeom g;
    load_xyz(args.bs, A, g.A);
    load_xyz(args.bs, B, g.B);
    load_xyz(args.bs, C, g.C);
    load_xyz(args.bs, D, g.D);

    // this lane's rows and units: offsets of their (a,b[,c]) slices in the 2D-integral arrays
    int rx[S::FR > 0 ? S::FR : 1], ry[S::FR > 0 ? S::FR : 1], rz[S::FR > 0 ? S::FR : 1];
#pragma unroll
    for (int k = 0; k < S::FR; ++k) {
        const int row = lane + G * k, a = row / NB, b = row - (row / NB) * NB;
        rx[k] = (cart_x(LA, a) * (LB + 1) + cart_x(LB, b)) * (LC + 1) * (LD + 1);
        ry[k] = (cart_y(LA, a) * (LB + 1) + cart_y(LB, b)) * (LC + 1) * (LD + 1);
        rz[k] = (cart_z(LA, a) * (LB + 1) + cart_z(LB, b)) * (LC + 1) * (LD + 1);
    }
    int ux[S::NU > 0 ? S::NU : 1], uy[S::NU > 0 ? S::NU : 1], uz[S::NU > 0 ? S::NU : 1];
#pragma unroll
    for (int j = 0; j < S::NU; ++j) {
        const int u = min(lane + G * j, S::NUNIT - 1);
        const int row = S::FR * G + u / NC, c = u % NC, a = row / NB, b = row % NB;
        ux[j] = ((cart_x(LA, a) * (LB + 1) + cart_x(LB, b)) * (LC + 1) + cart_x(LC, c)) * (LD + 1);
        uy[j] = ((cart_y(LA, a) * (LB + 1) + cart_y(LB, b)) * (LC + 1) + cart_y(LC, c)) * (LD + 1);
        uz[j] = ((cart_z(LA, a) * (LB + 1) + cart_z(LB, b)) * (LC + 1) + cart_z(LC, c)) * (LD + 1);
    }
    T accR[S::FR > 0 ? S::FR : 1][NCD], accU[S::NU > 0 ? S::NU : 1][ND];
#pragma unroll
    for (int k = 0; k < S::FR; ++k)
#pragma unroll
        for (int i = 0; i < NCD; ++i) accR[k][i] = T(0);
#pragma unroll
    for (int j = 0; j < S::NU; ++j)
#pragma unroll
        for (int i = 0; i < ND; ++i) accU[j][i] = T(0);

    const PrimPairs &pp = args.pp;
    const int pb0 = args.bra.poff[ib], npb = args.bra.np[ib], pk0 = args.ket.poff[ik], npk = args.ket.np[ik];
    for (int xb = pb0; xb < pb0 + npb; ++xb) {
        const double p = pp.a[xb] + pp.b[xb];
        const double Px = pp.Px[xb], Py = pp.Py[xb], Pz = pp.Pz[xb];
        const double Kb = pp.Kp[xb], argb = pp.arg[xb], hpb = pp.hp[xb];
        for (int xk = pk0; xk < pk0 + npk; ++xk) {
            if (argb + pp.arg[xk] > PDG_PRIMITIVE_CUT) continue;
            const double q = pp.a[xk] + pp.b[xk], hpk = pp.hp[xk];
            const double Qx = pp.Px[xk], Qy = pp.Py[xk], Qz = pp.Pz[xk];
            const double rs = rsqrt(p + q), rppq = rs * rs;
            const double PQx = Px - Qx, PQy = Py - Qy, PQz = Pz - Qz;
            const double x = p * q * rppq * (PQx * PQx + PQy * PQy + PQz * PQz);
            const double pref = TWO_PI_POW_2P5 * rs * Kb * pp.Kp[xk];
            __syncwarp(mask);  // the previous primitive's assembly has read the shared arrays
            for (int task = lane; task < 3 * NR; task += G) {
                const int r = task / 3, dir = task - 3 * (task / 3);
                double ur, wr;
                rys_root_single<NR>(x, r, ur, wr);
                ur *= rppq;
                const T b00 = T(0.5 * ur), b10 = T(hpb * (1.0 - q * ur)), b01 = T(hpk * (1.0 - p * ur));
                const double fq = q * ur, fp = p * ur;
                const double PA = dir == 0 ? Px - g.A[0] : dir == 1 ? Py - g.A[1] : Pz - g.A[2];
                const double QC = dir == 0 ? Qx - g.C[0] : dir == 1 ? Qy - g.C[1] : Qz - g.C[2];
                const double PQ = dir == 0 ? PQx : dir == 1 ? PQy : PQz;
                const double AB = dir == 0 ? g.A[0] - g.B[0] : dir == 1 ? g.A[1] - g.B[1] : g.A[2] - g.B[2];
                const double CD = dir == 0 ? g.C[0] - g.D[0] : dir == 1 ? g.C[1] - g.D[1] : g.C[2] - g.D[2];
                T Gm[LAB + 1][LCD + 1];
                rys_vrr<LAB, LCD, T>(Gm, T(dir == 2 ? wr * pref : 1.0), T(PA - fq * PQ), T(QC + fp * PQ), b10, b01, b00);
                hrr_store<LA, LB, LC, LD, T>(Gm, T(AB), T(CD), sI + task * NI);
            }
            __syncwarp(mask);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const T *__restrict__ Ix = sI + (3 * r) * NI;
                const T *__restrict__ Iy = Ix + NI;
                const T *__restrict__ Iz = Iy + NI;
#pragma unroll
                for (int k = 0; k < S::FR; ++k) {
                    T X[(LC + 1) * (LD + 1)], Y[(LC + 1) * (LD + 1)], Z[(LC + 1) * (LD + 1)];
#pragma unroll
                    for (int i = 0; i < (LC + 1) * (LD + 1); ++i) { X[i] = Ix[rx[k] + i]; Y[i] = Iy[ry[k] + i]; Z[i] = Iz[rz[k] + i]; }
#pragma unroll
                    for (int kc = 0; kc < NC; ++kc)
#pragma unroll
                        for (int ld = 0; ld < ND; ++ld)
                            accR[k][kc * ND + ld] += X[cart_x(LC, kc) * (LD + 1) + cart_x(LD, ld)] *
                                                     Y[cart_y(LC, kc) * (LD + 1) + cart_y(LD, ld)] *
                                                     Z[cart_z(LC, kc) * (LD + 1) + cart_z(LD, ld)];
                }
#pragma unroll
                for (int j = 0; j < S::NU; ++j) {
                    T X[LD + 1], Y[LD + 1], Z[LD + 1];
#pragma unroll
                    for (int i = 0; i <= LD; ++i) { X[i] = Ix[ux[j] + i]; Y[i] = Iy[uy[j] + i]; Z[i] = Iz[uz[j] + i]; }
#pragma unroll
                    for (int ld = 0; ld < ND; ++ld)
                        accU[j][ld] += X[cart_x(LD, ld)] * Y[cart_y(LD, ld)] * Z[cart_z(LD, ld)];
                }
            }
        }
    }
    __syncwarp(mask);
    // contracted block to shared memory, with the storage underflow
    const double uf = args.underflow;
#pragma unroll
    for (int k = 0; k < S::FR; ++k) {
        const int row = lane + G * k, a = row / NB, b = row - (row / NB) * NB;
        const double nab = comp_norm(LA, a) * comp_norm(LB, b);
#pragma unroll
        for (int kc = 0; kc < NC; ++kc)
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) {
                double v = (double)accR[k][kc * ND + ld];
                if (uf > 0.0 && fabs(v * nab * comp_norm(LC, kc) * comp_norm(LD, ld)) <= uf) v = 0.0;
                sm[row * NCDP + kc * ND + ld] = v;
            }
    }
#pragma unroll
    for (int j = 0; j < S::NU; ++j) {
        const int u = lane + G * j;
        if (u < S::NUNIT) {
            const int row = S::FR * G + u / NC, c = u % NC, a = row / NB, b = row % NB;
            const double nabc = comp_norm(LA, a) * comp_norm(LB, b) * comp_norm(LC, c);
#pragma unroll
            for (int ld = 0; ld < ND; ++ld) {
                double v = (double)accU[j][ld];
                if (uf > 0.0 && fabs(v * nabc * comp_norm(LD, ld)) <= uf) v = 0.0;
                sm[row * NCDP + c * ND + ld] = v;
            }
        }
    }
    // density blocks beside it: D_ab, D_cd, D_ac, D_ad, D_bc, D_bd
    const int n = args.n;
    const int oa = args.bs.sh_bf[A], ob = args.bs.sh_bf[B], oc = args.bs.sh_bf[C], od = args.bs.sh_bf[D];
    const double *__restrict__ Dm = args.D;
    double *dAB = sD, *dCD = dAB + NA * NB, *dAC = dCD + NC * ND, *dAD = dAC + NA * NC, *dBC = dAD + NA * ND,
           *dBD = dBC + NB * NC;
    for (int e = lane; e < NA * NB; e += G) dAB[e] = Dm[(oa + e / NB) * n + ob + e % NB];
    for (int e = lane; e < NC * ND; e += G) dCD[e] = Dm[(oc + e / ND) * n + od + e % ND];
    if (DOK) {
        for (int e = lane; e < NA * NC; e += G) dAC[e] = Dm[(oa + e / NC) * n + oc + e % NC];
        for (int e = lane; e < NA * ND; e += G) dAD[e] = Dm[(oa + e / ND) * n + od + e % ND];
        for (int e = lane; e < NB * NC; e += G) dBC[e] = Dm[(ob + e / NC) * n + oc + e % NC];
        for (int e = lane; e < NB * ND; e += G) dBD[e] = Dm[(ob + e / ND) * n + od + e % ND];
    }
    __syncwarp(mask);
    double s = 1.0;
    if (A == B) s *= 0.5;
    if (C == D) s *= 0.5;
    if (args.same && ib == ik) s *= 0.5;
    if (DOJ && scr.j) {
        const double s2 = 2.0 * s;
        for (int e = lane; e < NA * NB + NCD; e += G) {
            double acc = 0.0;
            if (e < NA * NB) {
#pragma unroll
                for (int cd = 0; cd < NCD; ++cd) acc += sm[e * NCDP + cd] * dCD[cd];
                atomicAdd(&args.J[(oa + e / NB) * n + ob + e % NB], s2 * acc);
            } else {
                const int cd = e - NA * NB;
#pragma unroll
                for (int ab = 0; ab < NA * NB; ++ab) acc += sm[ab * NCDP + cd] * dAB[ab];
                atomicAdd(&args.J[(oc + cd / ND) * n + od + cd % ND], s2 * acc);
            }
        }
    }
    if (DOK && scr.k) {
        constexpr int E1 = NA * NC, E2 = E1 + NA * ND, E3 = E2 + NB * NC, E4 = E3 + NB * ND;
        for (int e = lane; e < E4; e += G) {
            double acc = 0.0;
            if (e < E1) {  // Kt[a][c] += s sum_bd V D_bd
                const int a = e / NC, c = e % NC;
#pragma unroll
                for (int b = 0; b < NB; ++b)
#pragma unroll
                    for (int d = 0; d < ND; ++d) acc += sm[(a * NB + b) * NCDP + c * ND + d] * dBD[b * ND + d];
                atomicAdd(&args.K[(oa + a) * n + oc + c], s * acc);
            } else if (e < E2) {  // Kt[a][d] += s sum_bc V D_bc
                const int a = (e - E1) / ND, d = (e - E1) % ND;
#pragma unroll
                for (int b = 0; b < NB; ++b)
#pragma unroll
                    for (int c = 0; c < NC; ++c) acc += sm[(a * NB + b) * NCDP + c * ND + d] * dBC[b * NC + c];
                atomicAdd(&args.K[(oa + a) * n + od + d], s * acc);
            } else if (e < E3) {  // Kt[b][c] += s sum_ad V D_ad
                const int b = (e - E2) / NC, c = (e - E2) % NC;
#pragma unroll
                for (int a = 0; a < NA; ++a)
#pragma unroll
                    for (int d = 0; d < ND; ++d) acc += sm[(a * NB + b) * NCDP + c * ND + d] * dAD[a * ND + d];
                atomicAdd(&args.K[(ob + b) * n + oc + c], s * acc);
            } else {  // Kt[b][d] += s sum_ac V D_ac
                const int b = (e - E3) / ND, d = (e - E3) % ND;
#pragma unroll
                for (int a = 0; a < NA; ++a)
#pragma unroll
                    for (int c = 0; c < NC; ++c) acc += sm[(a * NB + b) * NCDP + c * ND + d] * dAC[a * NC + c];
                atomicAdd(&args.K[(ob + b) * n + od + d], s * acc);
            }
        }
    }
}

template <int LA, int LB, int LC, int LD, int G, bool DOJ, bool DOK, typename T>
void launch_jk_group(JKArgs a, const QuartetBlock &b, cudaStream_t st) {
    using S = GroupShape<LA, LB, LC, LD, G>;
    const size_t smem = (size_t)S::SMEM * S::GPB * sizeof(double);
    auto kern = eri_jk_group_kernel<LA, LB, LC, LD, G, DOJ, DOK, T>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int lanes[PDG_NBUCKET] = {G, G, G, G, G};
    const long long blocks = pdg_fill_work(a.work, b, lanes);
    { kern<<<(unsigned)blocks, 128, smem, st>>>(a); pdg_count_launch(); }
}

template <int CB, int CK, typename T>
void launch_jk_p(JKArgs a, const QuartetBlock &b, bool doJ, bool doK, cudaStream_t st) {
    constexpr int LA = PLA[CB], LB = PLB[CB], LC = PLA[CK], LD = PLB[CK];
    constexpr int G = jk_group(LA, LB, LC, LD);
    if constexpr (G > 0) {
        if (doJ && doK) launch_jk_group<LA, LB, LC, LD, G, true, true, T>(a, b, st);
        else if (doJ) launch_jk_group<LA, LB, LC, LD, G, true, false, T>(a, b, st);
        else launch_jk_group<LA, LB, LC, LD, G, false, true, T>(a, b, st);
    } else {
        const int v = a.variant >= 0 ? a.variant : jk_form(b);
        if (v == kWarpForm) {
            const long long blocks = pdg_fill_warp_work(a.work, b);
            if (doJ && doK) { eri_jk_warp_kernel<LA, LB, LC, LD, true, true, T><<<(unsigned)blocks, 128, 0, st>>>(a); pdg_count_launch(); }
            else if (doJ) { eri_jk_warp_kernel<LA, LB, LC, LD, true, false, T><<<(unsigned)blocks, 128, 0, st>>>(a); pdg_count_launch(); }
            else { eri_jk_warp_kernel<LA, LB, LC, LD, false, true, T><<<(unsigned)blocks, 128, 0, st>>>(a); pdg_count_launch(); }
            return;
        }
        const long long blocks = pdg_fill_work(a.work, b, jk_split(LA, LB, LC, LD) ? kSplitLanesV[v] : kWideLanes[v]);
        if (doJ && doK) { eri_jk_kernel<LA, LB, LC, LD, true, true, T><<<(unsigned)blocks, 128, 0, st>>>(a); pdg_count_launch(); }
        else if (doJ) { eri_jk_kernel<LA, LB, LC, LD, true, false, T><<<(unsigned)blocks, 128, 0, st>>>(a); pdg_count_launch(); }
        else { eri_jk_kernel<LA, LB, LC, LD, false, true, T><<<(unsigned)blocks, 128, 0, st>>>(a); pdg_count_launch(); }
    }
}

template <int CB, int CK>
void launch_jk_t(const JKArgs &a, const QuartetBlock &b, bool doJ, bool doK, bool fp32, cudaStream_t st) {
    if (fp32) launch_jk_p<CB, CK, float>(a, b, doJ, doK, st);
    else launch_jk_p<CB, CK, double>(a, b, doJ, doK, st);
}

}  // namespace

#define PDG_JK_ROW(cb, ...)                                     \
    const jk_launcher *pdg_jk_row##cb() {                       \
        static const jk_launcher row[PDG_NPAIRCLASS] = {__VA_ARGS__}; \
        return row;                                             \
    }
