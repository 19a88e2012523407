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
#include <cstring>
#include <string>
#include <atomic>
#include <type_traits>

#include "eri_jk.cuh"

std::atomic<int> pdg_jk_variant[PDG_NPAIRCLASS][PDG_NPAIRCLASS];

namespace {

// Schwarz bound per shell pair: Q = sqrt(max_ab |(ab|ab)|) with the true normalisation, eight lanes to a
// pair (one for d with d: one primitive pair).  Without the primitive-quartet cut, because a primitive pair
// cut in (ab|ab) can still contribute to (ab|cd) against a compact ket pair.  In one lane the 1296
// primitive quartets of two sixfold contracted s shells took 0.25 ms of every new geometry.
__host__ __device__ constexpr int schwarz_lanes(int la, int lb) { return la + lb < 4 ? 8 : 1; }

template <int LA, int LB>
__global__ void __launch_bounds__(64) schwarz_kernel(const int n, const int *__restrict__ shA,
                                                     const int *__restrict__ shB, const int *__restrict__ poff,
                                                     const int *__restrict__ np, PrimPairs pp, DeviceBasis bs,
                                                     double *__restrict__ Q) {
    constexpr int P = schwarz_lanes(LA, LB);
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) / P, lane = threadIdx.x & (P - 1);
    if (t >= n) return;
    constexpr int NA = ncart(LA), NB = ncart(LB);
    QuartetGeom g;
    load_xyz(bs, shA[t], g.A);
    load_xyz(bs, shB[t], g.B);
#pragma unroll
    for (int c = 0; c < 3; ++c) { g.C[c] = g.A[c]; g.D[c] = g.B[c]; }
    double V[NA * NB * NA * NB];
#pragma unroll
    for (int i = 0; i < NA * NB * NA * NB; ++i) V[i] = 0.0;
    const int p0 = poff[t], npr = np[t];
    for (int k = lane; k < npr * npr; k += P)
        eri_prim<LA, LB, LA, LB>(load_rec(pp.rec, p0 + k / npr), load_rec(pp.rec, p0 + k % npr), g, V);
    const unsigned mask = lane_group_mask(P);
    double m = 0.0;
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            double v = V[((a * NB + b) * NA + a) * NB + b];
#pragma unroll
            for (int o = P >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
            const double nn = comp_norm(LA, a) * comp_norm(LB, b);
            m = fmax(m, fabs(v) * nn * nn);
        }
    if (lane == 0) Q[t] = sqrt(m);
}

struct VariantInit {
    VariantInit() {
        for (int i = 0; i < PDG_NPAIRCLASS; ++i)
            for (int j = 0; j < PDG_NPAIRCLASS; ++j) pdg_jk_variant[i][j].store(-1);
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
    { schwarz_kernel<PLA[C], PLB[C]><<<(n * schwarz_lanes(PLA[C], PLB[C]) + 63) / 64, 64, 0, st>>>(n, shA, shB, poff, np, pp, bs, Q); pdg_count_launch(); }
}
typedef void (*schwarz_launcher)(int, const int *, const int *, const int *, const int *, const PrimPairs &,
                                 const DeviceBasis &, double *, cudaStream_t);
const schwarz_launcher schwarz_table[PDG_NPAIRCLASS] = {launch_schwarz_t<0>, launch_schwarz_t<1>, launch_schwarz_t<2>,
                                                        launch_schwarz_t<3>, launch_schwarz_t<4>, launch_schwarz_t<5>};

// Host arrays gathered for one transfer into one pool buffer: add() gives an array's place, send() copies all
// (stream-ordered on the context's non-blocking stream and complete on return).  The pool's buffer grows when
// needed and stays, so that a new geometry reuses the last one's.  A copy and its wait take some 10 us
// each, and the lists of a geometry are some 80 arrays.
class Staged {
    std::vector<char> bytes;

public:
    template <typename T>
    size_t add(const T *src, size_t n) {
        const size_t at = (bytes.size() + 15) / 16 * 16;
        bytes.resize(at + n * sizeof(T));
        if (n) std::memcpy(bytes.data() + at, src, n * sizeof(T));
        return at;
    }
    template <typename T>
    size_t add(const std::vector<T> &v) { return add(v.data(), v.size()); }
    int send(pdg_context *ctx, const char *name, char **dst) {
        *dst = (char *)pdg_pool(ctx, name, std::max<size_t>(16, bytes.size()));
        if (!*dst) { pdg_set_error("device buffer allocation failed (%s)", name); return PDG_ERR_ALLOC; }
        if (bytes.empty()) return PDG_OK;
        PDG_CUDA(cudaMemcpyAsync(*dst, bytes.data(), bytes.size(), cudaMemcpyHostToDevice, ctx->stream));
        PDG_CUDA(cudaStreamSynchronize(ctx->stream));
        return PDG_OK;
    }
};

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

// Exponent argument of a primitive pair, without fused operations: host and device count the same pairs.
__host__ __device__ __forceinline__ double primitive_arg(double ea, double eb, double r2) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(__ddiv_rn(__dmul_rn(ea, eb), __dadd_rn(ea, eb)), r2);
#else
    return ea * eb / (ea + eb) * r2;
#endif
}

// The primitive pairs of each shell pair (A, B, first primitive pair, squared distance), in the order the host
// counted them: one thread per shell pair.
__global__ void __launch_bounds__(128) pair_fill_kernel(int n, const int *__restrict__ shA, const int *__restrict__ shB,
                                                        const int *__restrict__ off, const double *__restrict__ dist2,
                                                        DeviceBasis bs, PrimPairs pp, double2 *__restrict__ rec,
                                                        float4 *__restrict__ rec32) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int A = shA[t], B = shB[t];
    double rA[3], rB[3];
    load_xyz(bs, A, rA);
    load_xyz(bs, B, rB);
    const double r2 = dist2[t];
    int i = off[t];
    for (int pa = bs.sh_poff[A]; pa < bs.sh_poff[A] + bs.sh_np[A]; ++pa) {
        const double ea = bs.prim_exp[pa], ca = bs.prim_coef[pa];
        for (int pb = bs.sh_poff[B]; pb < bs.sh_poff[B] + bs.sh_np[B]; ++pb) {
            const double eb = bs.prim_exp[pb], p = ea + eb, arg = primitive_arg(ea, eb, r2);
            if (arg > PDG_PRIMITIVE_CUT) continue;
            const double x = (ea * rA[0] + eb * rB[0]) / p, y = (ea * rA[1] + eb * rB[1]) / p, z = (ea * rA[2] + eb * rB[2]) / p;
            const double K = exp(-arg) * ca * bs.prim_coef[pb], Kp = K / p, hp = 0.5 / p;
            pp.a[i] = ea; pp.b[i] = eb;
            pp.Px[i] = x; pp.Py[i] = y; pp.Pz[i] = z;
            pp.K[i] = K; pp.arg[i] = arg; pp.Kp[i] = Kp; pp.hp[i] = hp;
            rec[4 * i] = make_double2(p, x); rec[4 * i + 1] = make_double2(y, z);
            rec[4 * i + 2] = make_double2(Kp, hp); rec[4 * i + 3] = make_double2(arg, ea);
            rec32[2 * i] = make_float4((float)p, (float)(x - rA[0]), (float)(y - rA[1]), (float)(z - rA[2]));
            rec32[2 * i + 1] = make_float4((float)Kp, (float)hp, (float)arg, 0.0f);
            ++i;
        }
    }
}

// Build primitive-pair data and Schwarz-sorted shell-pair lists for the current geometry.  The host counts
// the primitive pairs of each shell pair and sorts; the device forms them and the bounds, between two
// transfers up and one down (formed on the host and sent array by array, each waited for: 8 ms of a new
// geometry of 32 waters, 1.6 ms of one of 4).
static int build_pairs(pdg_context *ctx) {
    ProfScope prof(ctx, "pairs");
    const auto &sh = ctx->shells;
    const int ns = (int)sh.size();
    std::vector<int> cshA[PDG_NPAIRCLASS], cshB[PDG_NPAIRCLASS], cpoff[PDG_NPAIRCLASS], cnp[PDG_NPAIRCLASS];
    std::vector<double> cr2[PDG_NPAIRCLASS];
    int npp = 0;
    for (int i = 0; i < ns; ++i) {
        for (int j = 0; j <= i; ++j) {
            int A = i, B = j;
            if (sh[A].l < sh[B].l) std::swap(A, B);
            const double *rA = &ctx->xyz[3 * sh[A].atom], *rB = &ctx->xyz[3 * sh[B].atom];
            const double dx = rA[0] - rB[0], dy = rA[1] - rB[1], dz = rA[2] - rB[2];
            const double r2 = dx * dx + dy * dy + dz * dz;
            int cnt = 0;
            for (int pa = 0; pa < sh[A].np; ++pa)
                for (int pb = 0; pb < sh[B].np; ++pb)
                    cnt += !(primitive_arg(ctx->prim_exp[sh[A].poff + pa], ctx->prim_exp[sh[B].poff + pb], r2) > PDG_PRIMITIVE_CUT);
            if (cnt == 0) continue;
            const int c = pair_class(sh[A].l, sh[B].l);
            cshA[c].push_back(A);
            cshB[c].push_back(B);
            cpoff[c].push_back(npp);
            cnp[c].push_back(cnt);
            cr2[c].push_back(r2);
            npp += cnt;
        }
    }
    ctx->npp = npp;
    ctx->hostArg.clear();
    {
        const size_t n = std::max(1, npp);
        double *soa = (double *)pdg_pool(ctx, "pp.soa", 9 * n * sizeof(double));
        double2 *rec = (double2 *)pdg_pool(ctx, "pp.rec", 4 * n * sizeof(double2));
        float4 *rec32 = (float4 *)pdg_pool(ctx, "pp.rec32", 2 * n * sizeof(float4));
        if (!soa || !rec || !rec32) { pdg_set_error("device buffer allocation failed (primitive pairs)"); return PDG_ERR_ALLOC; }
        // the unsorted lists, all classes behind one another
        std::vector<int> A, B, O, N;
        std::vector<double> R;
        size_t first[PDG_NPAIRCLASS + 1] = {0};
        for (int c = 0; c < PDG_NPAIRCLASS; ++c) {
            A.insert(A.end(), cshA[c].begin(), cshA[c].end());
            B.insert(B.end(), cshB[c].begin(), cshB[c].end());
            O.insert(O.end(), cpoff[c].begin(), cpoff[c].end());
            N.insert(N.end(), cnp[c].begin(), cnp[c].end());
            R.insert(R.end(), cr2[c].begin(), cr2[c].end());
            first[c + 1] = A.size();
        }
        const int np = (int)A.size();
        Staged up;
        const size_t oA = up.add(A), oB = up.add(B), oO = up.add(O), oN = up.add(N), oR = up.add(R);
        char *d = nullptr;
        PDG_CHECK(up.send(ctx, "pairs.unsorted", &d));
        const int *dA = (const int *)(d + oA), *dB = (const int *)(d + oB), *dO = (const int *)(d + oO), *dN = (const int *)(d + oN);
        double *dQ = (double *)pdg_pool(ctx, "schwarz.Q", std::max(1, np) * sizeof(double));
        if (!dQ) { pdg_set_error("device buffer allocation failed (schwarz.Q)"); return PDG_ERR_ALLOC; }
        PrimPairs pp;
        double **arrays[] = {&pp.a, &pp.b, &pp.Px, &pp.Py, &pp.Pz, &pp.K, &pp.arg, &pp.Kp, &pp.hp};
        for (int k = 0; k < 9; ++k) *arrays[k] = soa + k * n;
        pp.rec = rec;
        pp.rec32 = rec32;
        std::vector<double> allQ(np);
        if (np > 0) {
            { pair_fill_kernel<<<(np + 127) / 128, 128, 0, ctx->stream>>>(np, dA, dB, dO, (const double *)(d + oR), ctx->dbasis, pp, rec, rec32); pdg_count_launch(); }
            {
                ClassFork fork(ctx);
                for (int c = 0; c < PDG_NPAIRCLASS; ++c)
                    schwarz_table[c]((int)(first[c + 1] - first[c]), dA + first[c], dB + first[c], dO + first[c], dN + first[c], pp,
                                     ctx->dbasis, dQ + first[c], fork.stream(1.0));
            }
            PDG_CUDA(cudaGetLastError());
            PDG_CUDA(cudaMemcpyAsync(allQ.data(), dQ, np * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
            PDG_CUDA(cudaStreamSynchronize(ctx->stream));
        }
        ctx->pp = pp;
        for (int c = 0; c < PDG_NPAIRCLASS; ++c) ctx->hostQ[c].assign(allQ.begin() + first[c], allQ.begin() + first[c + 1]);
    }
    // each class by primitive-count bucket, then by Schwarz bound (descending) inside a bucket
    Staged up;
    size_t at[PDG_NPAIRCLASS][6] = {};
    int ngroup[PDG_NPAIRCLASS] = {}, slots[PDG_NPAIRCLASS] = {};
    struct Key {
        double Q;
        int bucket, index;
    };
    std::vector<Key> key;
    for (int c = 0; c < PDG_NPAIRCLASS; ++c) {
        const int n = (int)cshA[c].size();
        ctx->bucket_start[c].assign(PDG_NBUCKET + 1, 0);
        ctx->qmax[c] = 0.0;
        ctx->hostPoff[c].resize(n);
        ctx->hostNp[c].resize(n);
        if (n == 0) continue;
        key.resize(n);
        for (int k = 0; k < n; ++k) key[k] = Key{ctx->hostQ[c][k] == ctx->hostQ[c][k] ? ctx->hostQ[c][k] : 0.0, np_bucket(cnp[c][k]), k};
        std::sort(key.begin(), key.end(), [](const Key &x, const Key &y) {
            return x.bucket != y.bucket ? x.bucket < y.bucket : x.Q != y.Q ? x.Q > y.Q : x.index < y.index;
        });
        std::vector<int> sA(n), sB(n);
        auto &sO = ctx->hostPoff[c], &sN = ctx->hostNp[c];
        auto &sQ = ctx->hostQ[c];
        for (int k = 0; k < n; ++k) {
            const int o = key[k].index;
            sA[k] = cshA[c][o]; sB[k] = cshB[c][o];
            sO[k] = cpoff[c][o]; sN[k] = cnp[c][o];
            sQ[k] = key[k].Q;
        }
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
        for (int kb = 0; kb < PDG_NBUCKET; ++kb) {
            bg[kb] = (int)goff.size();
            for (int k = bs[kb]; k < bs[kb + 1]; k += 32) {
                const int e = std::min(k + 32, bs[kb + 1]);
                goff.push_back(slots[c]);
                gfirst.push_back(k);
                gfirst.push_back(e - k);
                slots[c] += *std::max_element(sN.begin() + k, sN.begin() + e);
            }
        }
        ngroup[c] = (int)goff.size();
        if (ngroup[c] & 1) goff.push_back(0);  // the (first, count) pairs behind start on 8 bytes
        goff.insert(goff.end(), gfirst.begin(), gfirst.end());
        at[c][0] = up.add(sA); at[c][1] = up.add(sB); at[c][2] = up.add(sO);
        at[c][3] = up.add(sN); at[c][4] = up.add(sQ); at[c][5] = up.add(goff);
    }
    char *d = nullptr;
    PDG_CHECK(up.send(ctx, "pairs.lists", &d));
    for (int c = 0; c < PDG_NPAIRCLASS; ++c) {
        PairList &pl = ctx->pairs[c];
        pl.n = (int)cshA[c].size();
        if (pl.n == 0) continue;
        pl.shA = (int *)(d + at[c][0]);
        pl.shB = (int *)(d + at[c][1]);
        pl.poff = (int *)(d + at[c][2]);
        pl.np = (int *)(d + at[c][3]);
        pl.Q = (double *)(d + at[c][4]);
        const int *dg = (const int *)(d + at[c][5]);
        double2 *grec = (double2 *)pdg_pool(ctx, cname("pairs.grec", c).c_str(), (size_t)slots[c] * 128 * sizeof(double2));
        float4 *grec32 = (float4 *)pdg_pool(ctx, cname("pairs.grec32", c).c_str(), (size_t)slots[c] * 64 * sizeof(float4));
        if (!grec || !grec32) { pdg_set_error("device buffer allocation failed (pairs.grec)"); return PDG_ERR_ALLOC; }
        const int ng = ngroup[c];
        { ket_group_kernel<<<(ng + 3) / 4, 128, 0, ctx->stream>>>(ng, dg, reinterpret_cast<const int2 *>(dg + ng + (ng & 1)), pl, ctx->pp, grec, grec32); pdg_count_launch(); }
        PDG_CUDA(cudaGetLastError());
        pl.grec = grec;
        pl.grec32 = grec32;
        pl.goff = dg;
    }
    return PDG_OK;
}

// A failure part of the way (device memory) leaves no half of the lists: the next call starts over.
int pdg_ensure_pairs(pdg_context *ctx) {
    if (ctx->pp.a) return PDG_OK;
    const int status = build_pairs(ctx);
    if (status != PDG_OK) pdg_free_pairs(ctx);
    return status;
}

// One (bra class, ket class, ket bucket) of the work list while it is built.
struct BlockDesc {
    const double *need, *Qk;      // what a bra pair needs of a ket (threshold / its bound); bounds of the ket class
    const int *np;                // primitive pairs of the bra pairs
    int nb, k0, nk, same;
    long long *offs, *woffs;      // prefix sums over the bras (nb + 1 each)
    long long total, wtotal;      // quartets and (bra, ket group) items
    int *cbra, *wbra;             // their bra maps (bra_of)
};

// Prefix sums over the bra pairs of a bucket's surviving kets (pdg_ket_count) and of their groups of 32, with
// the totals and the bras' primitive pairs summed over the quartets: one CTA per descriptor.
__global__ void __launch_bounds__(1024) block_offsets_kernel(const BlockDesc *__restrict__ desc, long long *__restrict__ totals) {
    const BlockDesc b = desc[blockIdx.x];
    __shared__ long long ws[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long base = 0, wbase = 0, prims = 0;
    if (threadIdx.x == 0) b.offs[0] = b.woffs[0] = 0;
    for (int i0 = 0; i0 < b.nb; i0 += 1024) {
        const int i = i0 + threadIdx.x;
        long long cnt = 0;
        if (i < b.nb) {  // the bucket is sorted by Q descending: the kets with Q >= need are a prefix
            const double need = b.need[i];
            int lo = 0, hi = b.nk;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (b.Qk[b.k0 + mid] >= need) lo = mid + 1; else hi = mid;
            }
            cnt = lo;
            if (b.same) cnt = min(cnt, (long long)max(0, i - b.k0 + 1));
            prims += cnt * b.np[i];
        }
        long long s = cnt, g = (cnt + 31) / 32;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, s, o), v = __shfl_up_sync(0xffffffffu, g, o);
            if (lane >= o) { s += u; g += v; }
        }
        if (lane == 31) { ws[0][w] = s; ws[1][w] = g; }
        __syncthreads();
        if (w == 0) {
            long long x = ws[0][lane], y = ws[1][lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) { x += u; y += v; }
            }
            ws[0][lane] = x;
            ws[1][lane] = y;
        }
        __syncthreads();
        if (i < b.nb) {
            b.offs[i + 1] = base + s + (w ? ws[0][w - 1] : 0);
            b.woffs[i + 1] = wbase + g + (w ? ws[1][w - 1] : 0);
        }
        base += ws[0][31];
        wbase += ws[1][31];
        __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) prims += __shfl_xor_sync(0xffffffffu, prims, o);
    if (lane == 0) ws[0][w] = prims;
    __syncthreads();
    if (threadIdx.x == 0) {
        prims = 0;
        for (int k = 0; k < 32; ++k) prims += ws[0][k];
        totals[3 * blockIdx.x] = base;
        totals[3 * blockIdx.x + 1] = wbase;
        totals[3 * blockIdx.x + 2] = prims;
    }
}

// The bra maps: entry k = bra pair of item min(4k, total - 1) (binary search of the prefix sums), of the
// quartets (blockIdx.z 0) and of the (bra, ket group) items (1) of descriptor blockIdx.y.
__global__ void __launch_bounds__(256) bra_map_kernel(const BlockDesc *__restrict__ desc) {
    const BlockDesc b = desc[blockIdx.y];
    const long long *__restrict__ offs = blockIdx.z ? b.woffs : b.offs;
    const long long total = blockIdx.z ? b.wtotal : b.total;
    int *__restrict__ map = blockIdx.z ? b.wbra : b.cbra;
    const long long n = (total - 1) / 4 + 2;
    for (long long k = blockIdx.x * 256LL + threadIdx.x; k < n; k += gridDim.x * 256LL) {
        const long long t = min(4 * k, total - 1);
        int lo = 0, hi = b.nb;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (offs[mid] <= t) lo = mid; else hi = mid;
        }
        map[k] = lo;
    }
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
// in the class order (pdg_ket_count is the rule).
int pdg_build_blocks(pdg_context *ctx, double thr) {
    if (ctx->blocks_thr == thr && !ctx->blocks.empty()) return PDG_OK;
    ctx->blocks.clear();
    // what a bra needs of a ket, thr / Q_bra (infinite without a bound), by class
    Staged needs;
    size_t need_at[PDG_NPAIRCLASS] = {};
    std::vector<double> need;
    for (int c = 0; c < PDG_NPAIRCLASS; ++c) {
        need.resize(ctx->hostQ[c].size());
        for (size_t i = 0; i < need.size(); ++i) need[i] = ctx->hostQ[c][i] > 0.0 ? thr / ctx->hostQ[c][i] : HUGE_VAL;
        need_at[c] = needs.add(need);
    }
    struct Sub {
        int cb, ck, kb;
    };
    std::vector<Sub> subs;
    std::vector<BlockDesc> desc;
    size_t noffs = 0;
    for (int cb = 0; cb < PDG_NPAIRCLASS; ++cb) {
        const int nb = (int)ctx->hostQ[cb].size();
        if (nb == 0) continue;
        for (int ck = 0; ck <= cb; ++ck)
            for (int kb = 0; kb < PDG_NBUCKET; ++kb) {
                if (ctx->hostQ[ck].empty()) continue;
                const int k0 = ctx->bucket_start[ck][kb], nk = ctx->bucket_start[ck][kb + 1] - k0;
                if (nk <= 0) continue;
                subs.push_back(Sub{cb, ck, kb});
                desc.push_back(BlockDesc{nullptr, ctx->pairs[ck].Q, ctx->pairs[cb].np, nb, k0, nk, cb == ck, nullptr, nullptr, 0, 0, nullptr, nullptr});
                noffs += 2 * ((size_t)nb + 1);
            }
    }
    const int nsub = (int)subs.size();
    if (nsub == 0) { ctx->blocks_thr = thr; return PDG_OK; }
    long long *offs = (long long *)pdg_pool(ctx, "blocks.offs", noffs * sizeof(long long));
    long long *dtot = (long long *)pdg_pool(ctx, "blocks.totals", 3 * nsub * sizeof(long long));
    if (!offs || !dtot) { pdg_set_error("device buffer allocation failed (blocks.offs)"); return PDG_ERR_ALLOC; }
    char *dneed = nullptr, *ddesc = nullptr;
    PDG_CHECK(needs.send(ctx, "blocks.need", &dneed));
    for (int k = 0; k < nsub; ++k) {
        desc[k].need = (const double *)(dneed + need_at[subs[k].cb]);
        desc[k].offs = offs;
        desc[k].woffs = offs + desc[k].nb + 1;
        offs += 2 * ((size_t)desc[k].nb + 1);
    }
    {
        Staged up;
        up.add(desc);
        PDG_CHECK(up.send(ctx, "blocks.desc", &ddesc));
    }
    { block_offsets_kernel<<<nsub, 1024, 0, ctx->stream>>>((const BlockDesc *)ddesc, dtot); pdg_count_launch(); }
    PDG_CUDA(cudaGetLastError());
    std::vector<long long> tot(3 * nsub);
    PDG_CUDA(cudaMemcpyAsync(tot.data(), dtot, tot.size() * sizeof(long long), cudaMemcpyDeviceToHost, ctx->stream));
    PDG_CUDA(cudaStreamSynchronize(ctx->stream));
    // the bra maps of the lists that hold quartets
    std::vector<BlockDesc> live;
    size_t nmap = 0;
    long long longest = 0;
    for (int k = 0; k < nsub; ++k) {
        desc[k].total = tot[3 * k];
        desc[k].wtotal = tot[3 * k + 1];
        if (desc[k].total == 0) continue;
        nmap += (desc[k].total - 1) / 4 + 2 + (desc[k].wtotal - 1) / 4 + 2;
        longest = std::max(longest, desc[k].total);
    }
    int *map = (int *)pdg_pool(ctx, "blocks.maps", std::max<size_t>(1, nmap) * sizeof(int));
    if (!map) { pdg_set_error("device buffer allocation failed (blocks.maps)"); return PDG_ERR_ALLOC; }
    for (int k = 0; k < nsub; ++k) {
        BlockDesc &e = desc[k];
        if (e.total == 0) continue;
        e.cbra = map;
        e.wbra = e.cbra + ((e.total - 1) / 4 + 2);
        map = e.wbra + ((e.wtotal - 1) / 4 + 2);
        live.push_back(e);
        const Sub &u = subs[k];
        if (ctx->blocks.empty() || ctx->blocks.back().cb != u.cb || ctx->blocks.back().ck != u.ck) {
            QuartetBlock qb{};
            qb.cb = u.cb;
            qb.ck = u.ck;
            ctx->blocks.push_back(qb);
        }
        QuartetBlock &qb = ctx->blocks.back();
        auto &sb = qb.sub[qb.nsub++];
        sb.total = e.total;
        sb.wtotal = e.wtotal;
        sb.offs = e.offs;
        sb.woffs = e.woffs;
        sb.cbra = e.cbra;
        sb.wbra = e.wbra;
        sb.k0 = e.k0;
        sb.nk = e.nk;
        sb.bucket = u.kb;
        sb.g0 = ctx->bucket_group[u.ck][u.kb];
        qb.total += sb.total;
        const int lt = PLA[u.cb] + PLB[u.cb] + PLA[u.ck] + PLB[u.ck];
        const double per = 20.0 + (lt / 2 + 1) * ncart(PLA[u.cb]) * ncart(PLB[u.cb]) * ncart(PLA[u.ck]) * ncart(PLB[u.ck]);
        qb.cost += per * ctx->hostNp[u.ck][e.k0] * tot[3 * k + 2];
    }
    if (!live.empty()) {
        Staged up;
        up.add(live);
        PDG_CHECK(up.send(ctx, "blocks.desc", &ddesc));
        const unsigned gx = (unsigned)std::min<long long>(64, ((longest - 1) / 4 + 2 + 255) / 256);
        { bra_map_kernel<<<dim3(gx, (unsigned)live.size(), 2), 256, 0, ctx->stream>>>((const BlockDesc *)ddesc); pdg_count_launch(); }
        PDG_CUDA(cudaGetLastError());
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

// Tile autotuner of the kernels that split quartets over lanes: for every (bra class, ket class) work list of
// the current geometry that takes one of their tables (jk_form), time each table (one warm-up launch, then the
// best of two CUDA-event-timed launches of a full J+K build of the context's current density into scratch
// matrices) and keep the fastest, which every later list of the class pair below kWarpItems then takes, in
// every context of the process.  variants (36 ints, may be NULL) receives the choice per class pair (-1
// where nothing was tuned: no list, a longer list, or a class without tables to choose from).
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
        if (jk_group(la, lb, lc, ld) > 0 || !jk_split(la, lb, lc, ld) || jk_form(b) == kWarpForm) continue;
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
        int best = -1;
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

// What the next J/K build of the current lists launches for a class pair: a table of lanes, kWarpForm, or -1
// (no list, or the cooperative form).
extern "C" int pdg_jk_form_of(pdg_context *ctx, int cb, int ck) {
    if (!ctx || ctx->nbf == 0 || !ctx->have_geometry) return -1;
    if (pdg_ensure_pairs(ctx) != PDG_OK || pdg_build_blocks(ctx, ctx->schwarz_cut) != PDG_OK) return -1;
    for (const auto &b : ctx->blocks)
        if (b.cb == cb && b.ck == ck && jk_group(PLA[cb], PLB[cb], PLA[ck], PLB[ck]) == 0) return jk_form(b);
    return -1;
}
