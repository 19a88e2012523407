// Canonical purification of a small density in one launch (the iteration is described at purify_density).
//
// Step by step, a purification is two GEMMs and an update of a matrix that fits one SM's shared memory, some
// 20 to 40 times per SCF cycle: launches and the kernels' fixed times, about 8 us a step for 19 functions
// and 11 us for 100, are all of it.  Here a cluster of eight CTAs holds the iteration: each CTA keeps all of
// P and computes the columns of P^2 and P^3 = P P^2 that it owns (for P^3 it needs only those columns of
// P^2), the CTAs exchange the traces and the new columns over distributed shared memory, and two cluster
// barriers make a step: 2 us for 19 functions, 8 us for 110.
#include <cooperative_groups.h>

#include "context.h"

namespace cg = cooperative_groups;

namespace {

constexpr int PUR_CTAS = 8, PUR_T = 256;
constexpr int PUR_MMAX = 144;  // P (row stride 148) and the owned columns of P^2 fill 195 of 227 KB

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
// (the step taken then squares it) or after 120 steps.  RT row tiles of 8 per warp and CT column tiles per CTA
// cover 64 RT rows and 64 CT columns.
template <int RT, int CT>
__global__ void __cluster_dims__(PUR_CTAS, 1, 1) __launch_bounds__(PUR_T, 1)
    purify_cluster_kernel(int m, double *__restrict__ Q, double *__restrict__ status) {
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) double ps[];
    const int mp = pur_pad(m), ld = pur_ld(mp), nt = mp / 8, tpc = (nt + PUR_CTAS - 1) / PUR_CTAS;
    const int rank = (int)cluster.block_rank(), ct0 = rank * tpc, nc = max(0, min(tpc, nt - ct0));  // owned column tiles
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    double *P = ps, *P2 = ps + (size_t)mp * ld;  // P2[j][k]: owned column j of P^2
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
        double c2[RT][CT][2], c3[RT][CT][2];
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int c = 0; c < CT; ++c) c2[i][c][0] = c2[i][c][1] = c3[i][c][0] = c3[i][c][1] = 0.0;
        // P^2: P is symmetric, so that a column fragment is read as a row's
#pragma unroll 2
        for (int k = q; k < mp; k += 4) {
            double b[CT];
#pragma unroll
            for (int c = 0; c < CT; ++c) b[c] = c < nc ? P[(8 * (ct0 + c) + g) * ld + k] : 0.0;
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int rt = min(warp + 8 * i, nt - 1);  // a warp without a tile repeats the last one and drops it
                if (i > 0 && 8 * i >= nt) continue;
                const double a = P[(8 * rt + g) * ld + k];
#pragma unroll
                for (int c = 0; c < CT; ++c)
                    if (c < nc) dmma(c2[i][c][0], c2[i][c][1], a, b[c]);
            }
        }
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int c = 0; c < CT; ++c)
                if (warp + 8 * i < nt && c < nc) {
                    P2[(8 * c + 2 * q) * ld + 8 * (warp + 8 * i) + g] = c2[i][c][0];
                    P2[(8 * c + 2 * q + 1) * ld + 8 * (warp + 8 * i) + g] = c2[i][c][1];
                }
        __syncthreads();
#pragma unroll 2
        for (int k = q; k < mp; k += 4) {
            double b[CT];
#pragma unroll
            for (int c = 0; c < CT; ++c) b[c] = c < nc ? P2[(8 * c + g) * ld + k] : 0.0;
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int rt = min(warp + 8 * i, nt - 1);  // a warp without a tile repeats the last one and drops it
                if (i > 0 && 8 * i >= nt) continue;
                const double a = P[(8 * rt + g) * ld + k];
#pragma unroll
                for (int c = 0; c < CT; ++c)
                    if (c < nc) dmma(c3[i][c][0], c3[i][c][1], a, b[c]);
            }
        }
        // traces tr(P - P^2), tr(P^2 - P^3) of the owned columns, then of all, in the order of the ranks
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int c = 0; c < CT; ++c)
                if (c < nc && warp + 8 * i == ct0 + c && g >> 1 == q) {
                    const int d = 8 * (ct0 + c) + g;
                    const double p2 = g & 1 ? c2[i][c][1] : c2[i][c][0], p3 = g & 1 ? c3[i][c][1] : c3[i][c][0];
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
        // the owned columns of the new P over those of P^2, then, as rows, into every CTA's copy
        const double c = t1 / t0;
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int cc = 0; cc < CT; ++cc)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = 8 * (warp + 8 * i) + g, col = 8 * cc + 2 * q + e;
                    if (cc >= nc || row >= mp) continue;
                    const double p2 = c2[i][cc][e], p3 = c3[i][cc][e], p = P[(8 * ct0 + col) * ld + row];
                    P2[col * ld + row] = c >= 0.5 ? ((1.0 + c) * p2 - p3) / c : ((1.0 - 2.0 * c) * p + (1.0 + c) * p2 - p3) / (1.0 - c);
                }
        __syncthreads();
        for (int e = t; e < 8 * nc * (mp / 2); e += PUR_T) {
            const int row = e / (mp / 2), k = 2 * (e - row * (mp / 2));
            const double2 v = *reinterpret_cast<const double2 *>(&P2[row * ld + k]);
#pragma unroll
            for (int r = 0; r < PUR_CTAS; ++r)
                *reinterpret_cast<double2 *>(cluster.map_shared_rank(P, r) + (8 * ct0 + row) * ld + k) = v;
        }
        cluster.sync();
        if (fabs(t0) < 1e-12) break;
    }
    // (all CTAs leave the loop at the same step: they form t0 from the same numbers in the same order)
    for (int i = warp; i < m; i += PUR_T / 32)
        for (int j = 8 * ct0 + lane; j < min(m, 8 * (ct0 + nc)); j += 32) Q[(long long)i * m + j] = P[i * ld + j];
    if (rank == 0 && t == 0) status[0] = t0;
    cluster.sync();  // no CTA leaves while another may still write to it
}

}  // namespace

// Whether purify_cluster_kernel takes this size: all that its shared memory holds.  The GEMMs' steps grow
// slower with the size, but take 11 us at 110 functions.
bool pdg_purify_fits(int m) { return m <= PUR_MMAX; }

int pdg_purify_cluster(pdg_context *ctx, int m, double *d_Q, double *d_status) {
    const auto kern = m <= 64 ? purify_cluster_kernel<1, 1> : m <= 128 ? purify_cluster_kernel<2, 2> : purify_cluster_kernel<3, 3>;
    PDG_CUDA(pdg_allow_max_smem(kern));
    { kern<<<PUR_CTAS, PUR_T, pur_smem(m), ctx->stream>>>(m, d_Q, d_status); pdg_count_launch(); }
    PDG_CUDA(cudaGetLastError());
    return PDG_OK;
}
