// Integral-direct two-electron Coulomb/exchange build: Rys shell-quartet kernels grouped
// by angular-momentum class, Schwarz-screened, digested straight into J and K.
//
// Replaces the reference's stored-integral path: GaussianBasisContainerIntegrals_f2Cf2i
// (GaussianBases/__extensions__/csource/GaussianBasisContainerIntegrals_f2Xf2.c:74-139),
// GaussianBasisIntegrals_f2Cf2i (GaussianBasisIntegrals_f2Xf2.c:496-891) and the digest
// Fock_MakeFromTEIs / _Coulomb / _Exchange (QCModel/__extensions__/csource/FockConstruction.c:209-377).
//
#include <algorithm>
#include <cmath>
#include <numeric>
#include <string>
#include <atomic>
#include <type_traits>

#include "eri_jk.cuh"

std::atomic<int> pdg_jk_variant[PDG_NPAIRCLASS][PDG_NPAIRCLASS];

namespace {

// Schwarz bound per shell pair: Q = sqrt(max_ab |(ab|ab)|) with the true normalisation.
template <int LA, int LB>
__global__ void __launch_bounds__(64) schwarz_kernel(const int n, const int *__restrict__ shA,
                                                     const int *__restrict__ shB, const int *__restrict__ poff,
                                                     const int *__restrict__ np, PrimPairs pp, DeviceBasis bs,
                                                     double *__restrict__ Q) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    constexpr int NA = ncart(LA), NB = ncart(LB);
    QuartetGeom g;
    load_xyz(bs, shA[t], g.A);
    load_xyz(bs, shB[t], g.B);
#pragma unroll
    for (int c = 0; c < 3; ++c) { g.C[c] = g.A[c]; g.D[c] = g.B[c]; }
    double V[NA * NB * NA * NB];
    eri_block<LA, LB, LA, LB, false>(pp, poff[t], np[t], poff[t], np[t], g, V);
    double m = 0.0;
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const double nn = comp_norm(LA, a) * comp_norm(LB, b);
            m = fmax(m, fabs(V[((a * NB + b) * NA + a) * NB + b]) * nn * nn);
        }
    Q[t] = sqrt(m);
}

struct VariantInit {
    VariantInit() {
        for (int i = 0; i < PDG_NPAIRCLASS; ++i)
            for (int j = 0; j < PDG_NPAIRCLASS; ++j) pdg_jk_variant[i][j].store(kDefaultLanesV[i][j]);
    }
} g_variant_init;

jk_launcher jk_of(int cb, int ck) {
    const jk_launcher *const rows[PDG_NPAIRCLASS] = {pdg_jk_row0(), pdg_jk_row1(), pdg_jk_row2(),
                                                     pdg_jk_row3(), pdg_jk_row4(), pdg_jk_row5()};
    return rows[cb][ck];
}

template <int C>
void launch_schwarz_t(int n, const int *shA, const int *shB, const int *poff, const int *np, const PrimPairs &pp,
                      const DeviceBasis &bs, double *Q, cudaStream_t st) {
    if (n == 0) return;
    { schwarz_kernel<PLA[C], PLB[C]><<<(n + 63) / 64, 64, 0, st>>>(n, shA, shB, poff, np, pp, bs, Q); pdg_count_launch(); }
}
typedef void (*schwarz_launcher)(int, const int *, const int *, const int *, const int *, const PrimPairs &,
                                 const DeviceBasis &, double *, cudaStream_t);
const schwarz_launcher schwarz_table[PDG_NPAIRCLASS] = {launch_schwarz_t<0>, launch_schwarz_t<1>, launch_schwarz_t<2>,
                                                        launch_schwarz_t<3>, launch_schwarz_t<4>, launch_schwarz_t<5>};

// Upload into the context's named buffer pool (grown when needed, never freed before the context
// is destroyed), stream-ordered on the context's non-blocking stream and complete on return, so a
// new geometry reuses the device memory of the last one without allocating.
template <typename T>
int upload(pdg_context *ctx, const std::string &name, T **dst, const std::vector<T> &src) {
    *dst = (T *)pdg_pool(ctx, name.c_str(), std::max<size_t>(1, src.size()) * sizeof(T));
    if (!*dst) { pdg_set_error("device buffer allocation failed (%s)", name.c_str()); return PDG_ERR_ALLOC; }
    if (src.empty()) return PDG_OK;
    PDG_CUDA(cudaMemcpyAsync(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
    PDG_CUDA(cudaStreamSynchronize(ctx->stream));
    return PDG_OK;
}

std::string cname(const char *base, int c) { return std::string(base) + "." + std::to_string(c); }

}  // namespace

// The primitive records of a class's pairs in the group layout of PairList: one warp per group of 32
// pairs, one pair per lane (slots past a pair's own primitives are never read).
__global__ void __launch_bounds__(128) ket_group_kernel(int ng, const int *__restrict__ goff, const int2 *__restrict__ span,
                                                        PairList pl, PrimPairs pp, double2 *__restrict__ grec,
                                                        float4 *__restrict__ grec32) {
    const int g = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (g >= ng || lane >= span[g].y) return;
    const int k = span[g].x + lane, p0 = pl.poff[k], np = pl.np[k];
    for (int j = 0; j < np; ++j) {
        const size_t slot = (size_t)goff[g] + j;
        for (int f = 0; f < 4; ++f) grec[slot * 128 + 32 * f + lane] = pp.rec[4 * (p0 + j) + f];
        for (int f = 0; f < 2; ++f) grec32[slot * 64 + 32 * f + lane] = pp.rec32[2 * (p0 + j) + f];
    }
}

// Forget the shell-pair data of the last geometry; the device buffers stay in the context's pool.
void pdg_free_pairs(pdg_context *ctx) {
    for (int c = 0; c < PDG_NPAIRCLASS; ++c) ctx->pairs[c] = PairList{};
    ctx->pp = PrimPairs{};
    ctx->blocks.clear();
    ctx->blocks_thr = -1.0;
}

// Build primitive-pair data and Schwarz-sorted shell-pair lists for the current geometry.
int pdg_ensure_pairs(pdg_context *ctx) {
    if (ctx->pairs[0].shA || ctx->pp.a) return PDG_OK;
    ProfScope prof(ctx, "pairs");
    const auto &sh = ctx->shells;
    const int ns = (int)sh.size();
    std::vector<int> cshA[PDG_NPAIRCLASS], cshB[PDG_NPAIRCLASS], cpoff[PDG_NPAIRCLASS], cnp[PDG_NPAIRCLASS];
    std::vector<double> va, vb, vPx, vPy, vPz, vK, varg, vKp, vhp;
    std::vector<int> pair_atomA;   // atom of the first centre of each primitive pair
    for (int i = 0; i < ns; ++i) {
        for (int j = 0; j <= i; ++j) {
            int A = i, B = j;
            if (sh[A].l < sh[B].l) std::swap(A, B);
            const double *rA = &ctx->xyz[3 * sh[A].atom], *rB = &ctx->xyz[3 * sh[B].atom];
            const double dx = rA[0] - rB[0], dy = rA[1] - rB[1], dz = rA[2] - rB[2];
            const double r2 = dx * dx + dy * dy + dz * dz;
            const int off = (int)va.size();
            for (int pa = 0; pa < sh[A].np; ++pa) {
                const double ea = ctx->prim_exp[sh[A].poff + pa], ca = ctx->prim_coef[sh[A].poff + pa];
                for (int pb = 0; pb < sh[B].np; ++pb) {
                    const double eb = ctx->prim_exp[sh[B].poff + pb], cb = ctx->prim_coef[sh[B].poff + pb];
                    const double p = ea + eb;
                    const double arg = ea * eb / p * r2;
                    if (arg > PDG_PRIMITIVE_CUT) continue;
                    va.push_back(ea);
                    vb.push_back(eb);
                    vPx.push_back((ea * rA[0] + eb * rB[0]) / p);
                    vPy.push_back((ea * rA[1] + eb * rB[1]) / p);
                    vPz.push_back((ea * rA[2] + eb * rB[2]) / p);
                    vK.push_back(std::exp(-arg) * ca * cb);
                    varg.push_back(arg);
                    vKp.push_back(vK.back() / p);
                    vhp.push_back(0.5 / p);
                    pair_atomA.push_back(sh[A].atom);
                }
            }
            const int cnt = (int)va.size() - off;
            if (cnt == 0) continue;
            const int c = pair_class(sh[A].l, sh[B].l);
            cshA[c].push_back(A);
            cshB[c].push_back(B);
            cpoff[c].push_back(off);
            cnp[c].push_back(cnt);
        }
    }
    ctx->npp = (int)va.size();
    PDG_CHECK(upload(ctx, "pp.a", &ctx->pp.a, va));
    PDG_CHECK(upload(ctx, "pp.b", &ctx->pp.b, vb));
    PDG_CHECK(upload(ctx, "pp.Px", &ctx->pp.Px, vPx));
    PDG_CHECK(upload(ctx, "pp.Py", &ctx->pp.Py, vPy));
    PDG_CHECK(upload(ctx, "pp.Pz", &ctx->pp.Pz, vPz));
    PDG_CHECK(upload(ctx, "pp.K", &ctx->pp.K, vK));
    PDG_CHECK(upload(ctx, "pp.arg", &ctx->pp.arg, varg));
    PDG_CHECK(upload(ctx, "pp.Kp", &ctx->pp.Kp, vKp));
    PDG_CHECK(upload(ctx, "pp.hp", &ctx->pp.hp, vhp));
    {
        std::vector<double> rec(8 * va.size());
        for (size_t i = 0; i < va.size(); ++i) {
            double *r = &rec[8 * i];
            r[0] = va[i] + vb[i]; r[1] = vPx[i]; r[2] = vPy[i]; r[3] = vPz[i];
            r[4] = vKp[i]; r[5] = vhp[i]; r[6] = varg[i]; r[7] = va[i];
        }
        double *drec = nullptr;
        PDG_CHECK(upload(ctx, "pp.rec", &drec, rec));
        ctx->pp.rec = reinterpret_cast<const double2 *>(drec);
        std::vector<float> rec32(8 * va.size());
        for (size_t i = 0; i < va.size(); ++i) {
            float *r = &rec32[8 * i];
            const double *rA = &ctx->xyz[3 * pair_atomA[i]];
            r[0] = (float)(va[i] + vb[i]);
            r[1] = (float)(vPx[i] - rA[0]); r[2] = (float)(vPy[i] - rA[1]); r[3] = (float)(vPz[i] - rA[2]);
            r[4] = (float)vKp[i]; r[5] = (float)vhp[i]; r[6] = (float)varg[i]; r[7] = 0.0f;
        }
        float *drec32 = nullptr;
        PDG_CHECK(upload(ctx, "pp.rec32", &drec32, rec32));
        ctx->pp.rec32 = reinterpret_cast<const float4 *>(drec32);
    }
    ctx->hostArg = varg;
    // Schwarz bounds on the unsorted lists, then sort each class by Q descending.
    for (int c = 0; c < PDG_NPAIRCLASS; ++c) {
        const int n = (int)cshA[c].size();
        ctx->hostQ[c].clear();
        ctx->bucket_start[c].assign(PDG_NBUCKET + 1, 0);
        ctx->qmax[c] = 0.0;
        if (n == 0) continue;
        int *dA = nullptr, *dB = nullptr, *dO = nullptr, *dN = nullptr;
        double *dQ = nullptr;
        PDG_CHECK(upload(ctx, "schwarz.A", &dA, cshA[c]));
        PDG_CHECK(upload(ctx, "schwarz.B", &dB, cshB[c]));
        PDG_CHECK(upload(ctx, "schwarz.O", &dO, cpoff[c]));
        PDG_CHECK(upload(ctx, "schwarz.N", &dN, cnp[c]));
        dQ = (double *)pdg_pool(ctx, "schwarz.Q", n * sizeof(double));
        if (!dQ) { pdg_set_error("device buffer allocation failed (schwarz.Q)"); return PDG_ERR_ALLOC; }
        schwarz_table[c](n, dA, dB, dO, dN, ctx->pp, ctx->dbasis, dQ, ctx->stream);
        PDG_CUDA(cudaGetLastError());
        std::vector<double> Q(n);
        PDG_CUDA(cudaMemcpyAsync(Q.data(), dQ, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        PDG_CUDA(cudaStreamSynchronize(ctx->stream));
        // by primitive-count bucket, then by Schwarz bound (descending) inside a bucket
        std::vector<int> order(n);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
            const int bx = np_bucket(cnp[c][x]), by = np_bucket(cnp[c][y]);
            return bx != by ? bx < by : Q[x] > Q[y];
        });
        std::vector<int> sA(n), sB(n), sO(n), sN(n);
        std::vector<double> sQ(n);
        for (int k = 0; k < n; ++k) {
            sA[k] = cshA[c][order[k]]; sB[k] = cshB[c][order[k]];
            sO[k] = cpoff[c][order[k]]; sN[k] = cnp[c][order[k]];
            sQ[k] = Q[order[k]];
        }
        PairList &pl = ctx->pairs[c];
        pl.n = n;
        PDG_CHECK(upload(ctx, cname("pairs.shA", c), &pl.shA, sA));
        PDG_CHECK(upload(ctx, cname("pairs.shB", c), &pl.shB, sB));
        PDG_CHECK(upload(ctx, cname("pairs.poff", c), &pl.poff, sO));
        PDG_CHECK(upload(ctx, cname("pairs.np", c), &pl.np, sN));
        PDG_CHECK(upload(ctx, cname("pairs.Q", c), &pl.Q, sQ));
        ctx->hostQ[c] = sQ;
        ctx->hostPoff[c] = sO;
        ctx->hostNp[c] = sN;
        ctx->qmax[c] = *std::max_element(sQ.begin(), sQ.end());
        auto &bs = ctx->bucket_start[c];
        bs.assign(PDG_NBUCKET + 1, n);
        for (int k = n - 1; k >= 0; --k) bs[np_bucket(sN[k])] = k;
        for (int k = PDG_NBUCKET - 1; k >= 0; --k) bs[k] = std::min(bs[k], bs[k + 1]);
        // the pairs as kets in groups of 32 of a bucket, each group as many primitive slots as its
        // longest pair (PairList::grec)
        std::vector<int> goff, gfirst;  // first slot; first pair and pair count, by group
        auto &bg = ctx->bucket_group[c];
        bg.assign(PDG_NBUCKET, 0);
        int slots = 0;
        for (int kb = 0; kb < PDG_NBUCKET; ++kb) {
            bg[kb] = (int)goff.size();
            for (int k = bs[kb]; k < bs[kb + 1]; k += 32) {
                const int e = std::min(k + 32, bs[kb + 1]);
                goff.push_back(slots);
                gfirst.push_back(k);
                gfirst.push_back(e - k);
                slots += *std::max_element(sN.begin() + k, sN.begin() + e);
            }
        }
        const int ng = (int)goff.size();
        if (ng & 1) goff.push_back(0);  // the (first, count) pairs behind start on 8 bytes
        goff.insert(goff.end(), gfirst.begin(), gfirst.end());
        int *dg = nullptr;
        PDG_CHECK(upload(ctx, cname("pairs.goff", c), &dg, goff));
        double2 *grec = (double2 *)pdg_pool(ctx, cname("pairs.grec", c).c_str(), (size_t)slots * 128 * sizeof(double2));
        float4 *grec32 = (float4 *)pdg_pool(ctx, cname("pairs.grec32", c).c_str(), (size_t)slots * 64 * sizeof(float4));
        if (!grec || !grec32) { pdg_set_error("device buffer allocation failed (pairs.grec)"); return PDG_ERR_ALLOC; }
        { ket_group_kernel<<<(ng + 3) / 4, 128, 0, ctx->stream>>>(ng, dg, reinterpret_cast<const int2 *>(dg + ng + (ng & 1)), pl, ctx->pp, grec, grec32); pdg_count_launch(); }
        PDG_CUDA(cudaGetLastError());
        pl.grec = grec;
        pl.grec32 = grec32;
        pl.goff = dg;
    }
    return PDG_OK;
}

// cbra[k] = bra pair of quartet min(4k, total - 1) (binary search of the prefix sums).
__global__ void bra_map_kernel(const long long *__restrict__ offs, int nbra, long long total, long long nk,
                               int *__restrict__ cbra) {
    const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k >= nk) return;
    const long long t = min(4 * k, total - 1);
    int lo = 0, hi = nbra;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (offs[mid] <= t) lo = mid; else hi = mid;
    }
    cbra[k] = lo;
}

long long pdg_ket_count(const pdg_context *ctx, int cb, int ck, int ib, int k0, int nk, double thr) {
    const double qb = ctx->hostQ[cb][ib];
    if (!(qb > 0.0) || nk <= 0) return 0;
    const double need = thr / qb;
    const auto &Qk = ctx->hostQ[ck];
    // the bucket [k0, k0 + nk) is sorted by Q descending: the kets with Q >= need are a prefix
    long long cnt = std::upper_bound(Qk.begin() + k0, Qk.begin() + k0 + nk, need,
                                     [](double v, double e) { return v > e; }) - (Qk.begin() + k0);
    if (cb == ck) cnt = std::min<long long>(cnt, std::max<long long>(0, (long long)ib - k0 + 1));
    return cnt;
}

// Screened work list: for each (bra class >= ket class) block and each primitive-count bucket of the
// ket class, prefix sums over bra pairs of the number of ket pairs of the bucket with
// Q_bra * Q_ket >= thr; inside one class a quartet is counted once, with its ket at or before its bra
// in the class order.
int pdg_build_blocks(pdg_context *ctx, double thr) {
    if (ctx->blocks_thr == thr && !ctx->blocks.empty()) return PDG_OK;
    ctx->blocks.clear();
    int nbuf = 0;
    for (int cb = 0; cb < PDG_NPAIRCLASS; ++cb) {
        const auto &Qb = ctx->hostQ[cb];
        if (Qb.empty()) continue;
        for (int ck = 0; ck <= cb; ++ck) {
            if (ctx->hostQ[ck].empty()) continue;
            QuartetBlock qb{};
            qb.cb = cb;
            qb.ck = ck;
            const int lt = PLA[cb] + PLB[cb] + PLA[ck] + PLB[ck];
            const double per = 20.0 + (lt / 2 + 1) * ncart(PLA[cb]) * ncart(PLB[cb]) * ncart(PLA[ck]) * ncart(PLB[ck]);
            for (int kb = 0; kb < PDG_NBUCKET; ++kb) {
                const int k0 = ctx->bucket_start[ck][kb], nk = ctx->bucket_start[ck][kb + 1] - k0;
                if (nk <= 0) continue;
                // quartets, and behind them the (bra, group of 32 kets) items, as prefix sums over the bras
                const size_t nb = Qb.size();
                std::vector<long long> offs(2 * (nb + 1), 0);
                const double npk = ctx->hostNp[ck][k0];
                long long *woffs = &offs[nb + 1];
                for (size_t i = 0; i < nb; ++i) {
                    const long long cnt = pdg_ket_count(ctx, cb, ck, (int)i, k0, nk, thr);
                    offs[i + 1] = offs[i] + cnt;
                    woffs[i + 1] = woffs[i] + (cnt + 31) / 32;
                    qb.cost += per * npk * ctx->hostNp[cb][i] * cnt;
                }
                if (offs[nb] == 0) continue;
                auto &sb = qb.sub[qb.nsub++];
                sb.total = offs[nb];
                sb.wtotal = woffs[nb];
                sb.k0 = k0;
                sb.nk = nk;
                sb.bucket = kb;
                sb.g0 = ctx->bucket_group[ck][kb];
                PDG_CHECK(upload(ctx, cname("blocks.offs", nbuf), &sb.offs, offs));
                sb.woffs = sb.offs + nb + 1;
                const long long nmap = (sb.total - 1) / 4 + 2, wmap = (sb.wtotal - 1) / 4 + 2;
                sb.cbra = (int *)pdg_pool(ctx, cname("blocks.cbra", nbuf).c_str(), (nmap + wmap) * sizeof(int));
                if (!sb.cbra) { pdg_set_error("device buffer allocation failed (blocks.cbra)"); return PDG_ERR_ALLOC; }
                sb.wbra = sb.cbra + nmap;
                { bra_map_kernel<<<(unsigned)((nmap + 255) / 256), 256, 0, ctx->stream>>>(sb.offs, (int)nb, sb.total, nmap, sb.cbra); pdg_count_launch(); }
                { bra_map_kernel<<<(unsigned)((wmap + 255) / 256), 256, 0, ctx->stream>>>(sb.woffs, (int)nb, sb.wtotal, wmap, sb.wbra); pdg_count_launch(); }
                PDG_CUDA(cudaGetLastError());
                qb.total += sb.total;
                ++nbuf;
            }
            if (qb.nsub > 0) ctx->blocks.push_back(qb);
        }
    }
    // the launches overlap (ClassFork): the longest go first
    std::stable_sort(ctx->blocks.begin(), ctx->blocks.end(), [](const QuartetBlock &x, const QuartetBlock &y) { return x.cost > y.cost; });
    ctx->blocks_thr = thr;
    return PDG_OK;
}

// Largest |D'| over each shell-pair block (nshell x nshell, symmetric), for density screening.
__global__ void shell_pair_dmax_kernel(int ns, int n, const int *__restrict__ sh_bf, const int *__restrict__ sh_l,
                                       const double *__restrict__ D, double *__restrict__ dmax) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ns * ns) return;
    const int a = t / ns, b = t - a * ns;
    const int oa = sh_bf[a], ob = sh_bf[b], na = ncart(sh_l[a]), nb = ncart(sh_l[b]);
    double m = 0.0;
    for (int i = 0; i < na; ++i)
        for (int j = 0; j < nb; ++j) m = fmax(m, fabs(D[(long long)(oa + i) * n + ob + j]));
    dmax[t] = m;
}

int pdg_shell_pair_dmax(pdg_context *ctx, const double *d_D, double *d_dmax) {
    const int ns = (int)ctx->shells.size();
    { shell_pair_dmax_kernel<<<(ns * ns + 127) / 128, 128, 0, ctx->stream>>>(ns, ctx->nbf, ctx->dbasis.sh_bf, ctx->dbasis.sh_l, d_D, d_dmax); pdg_count_launch(); }
    PDG_CUDA(cudaGetLastError());
    return PDG_OK;
}

int pdg_eri_jk(pdg_context *ctx, const double *d_D, double *d_J, double *d_K, bool doJ, bool doK) {
    return pdg_eri_jk_screened(ctx, d_D, d_J, d_K, doJ, doK, nullptr, 0.0);
}

int pdg_eri_jk_screened(pdg_context *ctx, const double *d_D, double *d_J, double *d_K, bool doJ, bool doK,
                        const double *d_dmax, double dcut) {
    PDG_CHECK(pdg_ensure_pairs(ctx));
    PDG_CHECK(pdg_build_blocks(ctx, ctx->schwarz_cut));
    const bool mixed = ctx->precision_mode == 1;
    const int ns = (int)ctx->shells.size();
    if (mixed && !d_dmax) {
        // the precision partition needs the density bound even without density screening
        double *dm = (double *)pdg_pool(ctx, "jk_dmax", (size_t)ns * ns * sizeof(double));
        if (!dm) { pdg_set_error("pdg_eri_jk: device buffer allocation failed"); return PDG_ERR_ALLOC; }
        PDG_CHECK(pdg_shell_pair_dmax(ctx, d_D, dm));
        d_dmax = dm;
        dcut = 0.0;
    }
    if (mixed && !ctx->d_count32) {
        ctx->d_count32 = (unsigned long long *)pdg_pool(ctx, "count32", sizeof(unsigned long long));
        if (!ctx->d_count32) { pdg_set_error("pdg_eri_jk: device buffer allocation failed"); return PDG_ERR_ALLOC; }
        PDG_CUDA(cudaMemsetAsync(ctx->d_count32, 0, sizeof(unsigned long long), ctx->stream));
    }
    long long nq = 0;
    ProfScope prof(ctx, "eri_jk");
    ClassFork fork(ctx);
    for (const auto &b : ctx->blocks) {
        JKArgs a;
        a.bra = ctx->pairs[b.cb];
        a.ket = ctx->pairs[b.ck];
        a.same = (b.cb == b.ck);
        a.pp = ctx->pp;
        a.bs = ctx->dbasis;
        a.D = d_D;
        a.J = d_J;
        a.K = d_K;
        a.n = ctx->nbf;
        a.underflow = ctx->tei_underflow;
        a.dmax = d_dmax;
        a.nshell = ns;
        a.dcut = dcut;
        a.mixed_cut = ctx->mixed_cut;
        a.count32 = ctx->d_count32;
        a.variant = -1;
        if (mixed) {
            // quartets whose bound Q_AB Q_CD max|D| is below mixed_cut in FP32, the rest in FP64
            a.part = 1;
            jk_of(b.cb, b.ck)(a, b, doJ, doK, false, fork.stream(b.cost));
            PDG_CUDA(cudaGetLastError());
            a.part = 2;
            jk_of(b.cb, b.ck)(a, b, doJ, doK, true, fork.stream(b.cost));
        } else {
            a.part = 0;
            jk_of(b.cb, b.ck)(a, b, doJ, doK, false, fork.stream(b.cost));
        }
        PDG_CUDA(cudaGetLastError());
        nq += b.total;
    }
    ctx->last_quartets = nq;
    return PDG_OK;
}

// Tile autotuner of the one-thread J+K kernels: for every (bra class, ket class) work list of the
// current geometry whose kernel splits quartets over lanes, time each candidate lanes-per-bucket
// table (one warm-up launch, then the best of two CUDA-event-timed launches of a full J+K build of
// the context's current density into scratch matrices) and keep the fastest in the process-wide
// table every later build of every context uses.  variants (36 ints, may be NULL) receives the
// choice per class pair (-1 where nothing was tuned).
extern "C" int pdg_autotune_eri(pdg_context *ctx, int *variants) {
    if (!ctx) { pdg_set_error("pdg_autotune_eri: invalid argument"); return PDG_ERR_ARG; }
    if (ctx->nbf == 0 || !ctx->have_geometry) { pdg_set_error("pdg_autotune_eri: basis and geometry required"); return PDG_ERR_STATE; }
    cudaSetDevice(ctx->device);
    PDG_CHECK(pdg_ensure_pairs(ctx));
    PDG_CHECK(pdg_build_blocks(ctx, ctx->schwarz_cut));
    const size_t nn = (size_t)ctx->nbf * ctx->nbf * sizeof(double);
    double *J = (double *)pdg_pool(ctx, "tune.J", nn), *K = (double *)pdg_pool(ctx, "tune.K", nn);
    if (!J || !K) { pdg_set_error("pdg_autotune_eri: device buffer allocation failed"); return PDG_ERR_ALLOC; }
    if (variants)
        for (int k = 0; k < PDG_NPAIRCLASS * PDG_NPAIRCLASS; ++k) variants[k] = -1;
    cudaEvent_t e0, e1;
    PDG_CUDA(cudaEventCreate(&e0));
    PDG_CUDA(cudaEventCreate(&e1));
    int status = PDG_OK;
    for (const auto &b : ctx->blocks) {
        const int la = PLA[b.cb], lb = PLB[b.cb], lc = PLA[b.ck], ld = PLB[b.ck];
        if (jk_group(la, lb, lc, ld) > 0 || !jk_split(la, lb, lc, ld)) continue;
        JKArgs a;
        a.bra = ctx->pairs[b.cb];
        a.ket = ctx->pairs[b.ck];
        a.same = (b.cb == b.ck);
        a.pp = ctx->pp;
        a.bs = ctx->dbasis;
        a.D = ctx->d_D;
        a.J = J;
        a.K = K;
        a.n = ctx->nbf;
        a.underflow = ctx->tei_underflow;
        a.dmax = nullptr;
        a.nshell = (int)ctx->shells.size();
        a.dcut = 0.0;
        a.mixed_cut = ctx->mixed_cut;
        a.count32 = nullptr;
        a.part = 0;
        int best = kDefaultLanesV[b.cb][b.ck];
        float best_ms = 1e30f;
        for (int v = 0; v < kNLanesV && status == PDG_OK; ++v) {
            a.variant = v;
            float ms_v = 1e30f;
            for (int rep = 0; rep < 3; ++rep) {
                cudaEventRecord(e0, ctx->stream);
                jk_of(b.cb, b.ck)(a, b, true, true, false, ctx->stream);
                cudaEventRecord(e1, ctx->stream);
                if (cudaEventSynchronize(e1) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
                    pdg_set_error("pdg_autotune_eri: a timed launch failed");
                    status = PDG_ERR_CUDA;
                    break;
                }
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, e0, e1);
                if (rep > 0 && ms < ms_v) ms_v = ms;
            }
            if (ms_v < best_ms) { best_ms = ms_v; best = v; }
        }
        if (status != PDG_OK) break;
        pdg_jk_variant[b.cb][b.ck].store(best);
        if (variants) variants[b.cb * PDG_NPAIRCLASS + b.ck] = best;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return status;
}
