// Canonical purification of a small density in one launch (the iteration is described at purify_density).
//
// Step by step, a purification is two GEMMs and an update of a matrix that fits one SM's shared memory, some
// 20 to 40 times per SCF cycle: launches and the kernels' fixed times, 14 us a step for 19 functions and
// 18 us for 110, are all of it.  Here a cluster of eight CTAs holds the iteration: each CTA keeps all of
// P and computes the rows of P^2 and P^3 = P^2 P that it owns (for P^3 it needs only those rows of
// P^2), the CTAs exchange the traces and the new rows over distributed shared memory, and two cluster
// barriers make a step: 2.8 us for 19 functions, 11 us for 110.
#include <cooperative_groups.h>

#include "context.h"

namespace cg = cooperative_groups;

namespace {

constexpr int PUR_CTAS = 8, PUR_T = 256;
// At 128 functions a step takes 12 us here, 18 us as GEMMs; at 129 (three tiles per warp) 22 us against 20 us.
// P (row stride 132) and the owned rows of P^2 fill 149 KB.
constexpr int PUR_MMAX = 128;

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// Padded size and row stride (4 mod 16 doubles: a fragment's rows land in distinct banks).
__host__ __device__ constexpr int pur_pad(int m) { return (m + 7) / 8 * 8; }
__host__ __device__ constexpr int pur_ld(int mp) { return mp % 16 == 0 ? mp + 4 : mp + 12; }
inline size_t pur_smem(int m) {
    const int mp = pur_pad(m), tpc = (mp / 8 + PUR_CTAS - 1) / PUR_CTAS;
    return ((size_t)(mp + 8 * tpc) * pur_ld(mp) + 4 * PUR_CTAS + 2 * (PUR_T / 32)) * sizeof(double);
}

// Q (m x m): P0 in, the projector out; status[0] = the last tr(P - P^2).  Stops once that is below 1e-12
// (the step taken then squares it) or after 120 steps.  CT column tiles of 8 per warp and RT row tiles per CTA
// cover 64 CT columns and 64 RT rows.
//
// The products are P P and (P P) P of P as it is, not P P^T, although P is symmetric but for rounding: only
// these cancel its antisymmetric part K.  With P P^T (columns read as rows), P^3 and the rounding of X^T F X
// make a K that a step near the projector multiplies by up to 1/c <= 2 and the traces do not see: 2e-8 in
// the projector of a C, N, O molecule of 95 functions in PBE, 40 steps; so 1e-14, in the same time.
template <int CT, int RT>
__global__ void __cluster_dims__(PUR_CTAS, 1, 1) __launch_bounds__(PUR_T, 1)
    purify_cluster_kernel(int m, double *__restrict__ Q, double *__restrict__ status) {
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) double ps[];
    const int mp = pur_pad(m), ld = pur_ld(mp), nt = mp / 8, tpc = (nt + PUR_CTAS - 1) / PUR_CTAS;
    const int rank = (int)cluster.block_rank(), rt0 = rank * tpc, nr = max(0, min(tpc, nt - rt0));  // owned row tiles
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    double *P = ps, *P2 = ps + (size_t)mp * ld;  // P2[r][k]: owned row r of P^2
    // the CTAs' traces, two steps of them, and the warps'
    double (*part)[PUR_CTAS][2] = reinterpret_cast<double (*)[PUR_CTAS][2]>(P2 + (size_t)8 * tpc * ld);
    double (*wred)[2] = reinterpret_cast<double (*)[2]>(part + 2);
    for (int e = t; e < mp * mp; e += PUR_T) {
        const int i = e / mp, j = e - i * mp;
        P[i * ld + j] = i < m && j < m ? Q[(long long)i * m + j] : 0.0;
    }
    double t0 = 0.0;
    cluster.sync();
    for (int it = 0; it < 120; ++it) {
        double c2[CT][RT][2], c3[CT][RT][2];
#pragma unroll
        for (int i = 0; i < CT; ++i)
#pragma unroll
            for (int r = 0; r < RT; ++r) c2[i][r][0] = c2[i][r][1] = c3[i][r][0] = c3[i][r][1] = 0.0;
        // owned rows of P^2; with the stride, a half warp's column fragment falls into distinct banks too
#pragma unroll 2
        for (int k = q; k < mp; k += 4) {
            double a[RT];
#pragma unroll
            for (int r = 0; r < RT; ++r) a[r] = r < nr ? P[(8 * (rt0 + r) + g) * ld + k] : 0.0;
#pragma unroll
            for (int i = 0; i < CT; ++i) {
                const int ct = min(warp + 8 * i, nt - 1);  // a warp without a tile repeats the last one and drops it
                if (i > 0 && 8 * i >= nt) continue;
                const double b = P[k * ld + 8 * ct + g];
#pragma unroll
                for (int r = 0; r < RT; ++r)
                    if (r < nr) dmma(c2[i][r][0], c2[i][r][1], a[r], b);
            }
        }
#pragma unroll
        for (int i = 0; i < CT; ++i)
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (warp + 8 * i < nt && r < nr)
                    *reinterpret_cast<double2 *>(&P2[(8 * r + g) * ld + 8 * (warp + 8 * i) + 2 * q]) = make_double2(c2[i][r][0], c2[i][r][1]);
        __syncthreads();
#pragma unroll 2
        for (int k = q; k < mp; k += 4) {
            double a[RT];
#pragma unroll
            for (int r = 0; r < RT; ++r) a[r] = r < nr ? P2[(8 * r + g) * ld + k] : 0.0;
#pragma unroll
            for (int i = 0; i < CT; ++i) {
                const int ct = min(warp + 8 * i, nt - 1);  // a warp without a tile repeats the last one and drops it
                if (i > 0 && 8 * i >= nt) continue;
                const double b = P[k * ld + 8 * ct + g];
#pragma unroll
                for (int r = 0; r < RT; ++r)
                    if (r < nr) dmma(c3[i][r][0], c3[i][r][1], a[r], b);
            }
        }
        // traces tr(P - P^2), tr(P^2 - P^3) of the owned rows, then of all, in the order of the ranks
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int i = 0; i < CT; ++i)
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (r < nr && warp + 8 * i == rt0 + r && g >> 1 == q) {
                    const int d = 8 * (rt0 + r) + g;
                    const double p2 = g & 1 ? c2[i][r][1] : c2[i][r][0], p3 = g & 1 ? c3[i][r][1] : c3[i][r][0];
                    x += P[d * ld + d] - p2;
                    y += p2 - p3;
                }
        x = warp_sum(x);
        y = warp_sum(y);
        if (lane == 0) { wred[warp][0] = x; wred[warp][1] = y; }
        __syncthreads();
        if (t < PUR_CTAS) {
            double sx = 0.0, sy = 0.0;
            for (int w = 0; w < PUR_T / 32; ++w) { sx += wred[w][0]; sy += wred[w][1]; }
            double *o = cluster.map_shared_rank(&part[it & 1][rank][0], t);
            o[0] = sx;
            o[1] = sy;
        }
        cluster.sync();  // the traces are there, and no CTA reads P as an operand any more
        t0 = 0.0;
        double t1 = 0.0;
#pragma unroll
        for (int r = 0; r < PUR_CTAS; ++r) { t0 += part[it & 1][r][0]; t1 += part[it & 1][r][1]; }
        if (!(fabs(t0) > 1e-300)) break;  // already idempotent
        // the owned rows of the new P over those of P^2, then into every CTA's copy
        const double c = t1 / t0;
#pragma unroll
        for (int i = 0; i < CT; ++i)
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                if (rr >= nr || warp + 8 * i >= nt) continue;
                const int col = 8 * (warp + 8 * i) + 2 * q;
                const double2 p = *reinterpret_cast<const double2 *>(&P[(8 * (rt0 + rr) + g) * ld + col]);
                double v[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double p1 = e ? p.y : p.x, p2 = c2[i][rr][e], p3 = c3[i][rr][e];
                    v[e] = c >= 0.5 ? ((1.0 + c) * p2 - p3) / c : ((1.0 - 2.0 * c) * p1 + (1.0 + c) * p2 - p3) / (1.0 - c);
                }
                *reinterpret_cast<double2 *>(&P2[(8 * rr + g) * ld + col]) = make_double2(v[0], v[1]);
            }
        __syncthreads();
        for (int e = t; e < 8 * nr * (mp / 2); e += PUR_T) {
            const int row = e / (mp / 2), k = 2 * (e - row * (mp / 2));
            const double2 v = *reinterpret_cast<const double2 *>(&P2[row * ld + k]);
#pragma unroll
            for (int r = 0; r < PUR_CTAS; ++r)
                *reinterpret_cast<double2 *>(cluster.map_shared_rank(P, r) + (8 * rt0 + row) * ld + k) = v;
        }
        cluster.sync();
        if (fabs(t0) < 1e-12) break;
    }
    // (all CTAs leave the loop at the same step: they form t0 from the same numbers in the same order)
    for (int i = 8 * rt0 + warp; i < min(m, 8 * (rt0 + nr)); i += PUR_T / 32)
        for (int j = lane; j < m; j += 32) Q[(long long)i * m + j] = P[i * ld + j];
    if (rank == 0 && t == 0) status[0] = t0;
    cluster.sync();  // no CTA leaves while another may still write to it
}

}  // namespace

namespace {

using PurifyKernel = void (*)(int, double *, double *);
PurifyKernel purify_kernel(int m) { return m <= 64 ? purify_cluster_kernel<1, 1> : purify_cluster_kernel<2, 2>; }

}  // namespace

// How many clusters of the one-launch form for m functions the current device holds at a time; 0 above
// PUR_MMAX, and where eight such CTAs have no place together (a partitioned device, none at all).
extern "C" int pdg_purify_clusters(int m) {
    if (m < 1 || m > PUR_MMAX) return 0;
    const PurifyKernel kern = purify_kernel(m);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute dims[1];
    dims[0].id = cudaLaunchAttributeClusterDimension;
    dims[0].val.clusterDim.x = PUR_CTAS;
    dims[0].val.clusterDim.y = dims[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(PUR_CTAS);
    cfg.blockDim = dim3(PUR_T);
    cfg.dynamicSmemBytes = pur_smem(m);
    cfg.attrs = dims;
    cfg.numAttrs = 1;
    int n = 0;
    if (pdg_allow_max_smem(kern) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// Whether purify_cluster_kernel takes this size on the context's device (asked once per kernel, for its largest
// size).
bool pdg_purify_fits(pdg_context *ctx, int m) {
    if (m > PUR_MMAX) return false;
    int &n = ctx->purify_clusters[m <= 64 ? 0 : 1];
    if (n < 0) n = pdg_purify_clusters(m <= 64 ? 64 : PUR_MMAX);
    return n > 0;
}

int pdg_purify_cluster(pdg_context *ctx, int m, double *d_Q, double *d_status) {
    const PurifyKernel kern = purify_kernel(m);
    PDG_CUDA(pdg_allow_max_smem(kern));
    { kern<<<PUR_CTAS, PUR_T, pur_smem(m), ctx->stream>>>(m, d_Q, d_status); pdg_count_launch(); }
    PDG_CUDA(cudaGetLastError());
    return PDG_OK;
}
