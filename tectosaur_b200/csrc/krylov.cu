// One Arnoldi step of the constrained solve (examples/solve.py:25-61 runs
// scipy's GMRES on the host): classical Gram-Schmidt applied twice against the
// basis, the norm and the next basis vector, in one launch of an 8-CTA cluster.
//
// At the sizes of the plain solve (some thousand unknowns, tens of basis
// vectors: a few MB) the step is bound by launches, not by bytes: the products
// against the basis, their subtractions, the norm and the scaling took eleven
// launches.  Every CTA keeps its slice of w in shared memory; the slices' dot
// products are exchanged through distributed shared memory and added in rank
// order (deterministic), with the hardware's cluster barrier between phases.
// One cluster reads about 1 TB/s from L2, so larger steps stay with the
// library's matrix-vector products (tct_arnoldi_step_fits: above 1.5e6 basis
// entries the four passes would take longer than eleven launches).
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace tct {
namespace {

constexpr int ARN_CTAS = 8, ARN_THREADS = 512;
constexpr int ARN_SLICE = 4096;   // unknowns per CTA
constexpr int ARN_ROWS = 1024;    // basis vectors
constexpr int64_t ARN_WORK = 1500000;

constexpr size_t ARN_SMEM = sizeof(double) * (ARN_SLICE + 4 * ARN_ROWS);

__global__ void __cluster_dims__(ARN_CTAS, 1, 1) __launch_bounds__(ARN_THREADS)
arnoldi_kernel(double* __restrict__ V, int64_t n, int rows, const double* __restrict__ w,
               double* __restrict__ col) {
    extern __shared__ double sh[];
    double* ws = sh;                    // slice of w
    double* part1 = ws + ARN_SLICE;     // dot products of the slice, both sweeps
    double* part2 = part1 + ARN_ROWS;
    double* h1 = part2 + ARN_ROWS;      // their sums over the cluster
    double* h2 = h1 + ARN_ROWS;
    __shared__ double wsum[ARN_THREADS / 32], norm_part;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t per = (n + ARN_CTAS - 1) / ARN_CTAS;
    const int64_t s0 = min(n, rank * per);
    const int len = (int)(min(n, s0 + per) - s0);
    const double* Vs = V + s0;

    auto warp_sum = [](double s) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    // part[i] = V_i . ws over the slice, then h[i] = the cluster's sum
    auto project = [&](double* part, double* h) {
        for (int i = warp; i < rows; i += ARN_THREADS / 32) {
            const double* v = Vs + i * n;
            double s = 0;
            for (int k = lane; k < len; k += 32) s += v[k] * ws[k];
            s = warp_sum(s);
            if (lane == 0) part[i] = s;
        }
        cl.sync();
        for (int i = tid; i < rows; i += ARN_THREADS) {
            double s = 0;
#pragma unroll
            for (int c = 0; c < ARN_CTAS; c++) s += cl.map_shared_rank(part, c)[i];
            h[i] = s;
        }
        __syncthreads();
    };
    auto subtract = [&](const double* h) {
        for (int k = tid; k < len; k += ARN_THREADS) {
            double s = 0;
#pragma unroll 8
            for (int i = 0; i < rows; i++) s += h[i] * Vs[i * n + k];
            ws[k] -= s;
        }
        __syncthreads();
    };

    for (int k = tid; k < len; k += ARN_THREADS) ws[k] = w[s0 + k];
    __syncthreads();
    project(part1, h1);
    subtract(h1);
    project(part2, h2);
    subtract(h2);
    double s = 0;
    for (int k = tid; k < len; k += ARN_THREADS) s += ws[k] * ws[k];
    s = warp_sum(s);
    if (lane == 0) wsum[warp] = s;
    __syncthreads();
    if (tid == 0) {
        double t = 0;
        for (int i = 0; i < ARN_THREADS / 32; i++) t += wsum[i];
        norm_part = t;
    }
    cl.sync();
    double nn = 0;
#pragma unroll
    for (int c = 0; c < ARN_CTAS; c++) nn += *cl.map_shared_rank(&norm_part, c);
    nn = sqrt(nn);
    if (nn > 0.0)
        for (int k = tid; k < len; k += ARN_THREADS) V[rows * n + s0 + k] = ws[k] / nn;
    if (rank == 0) {
        for (int i = tid; i < rows; i += ARN_THREADS) col[i] = h1[i] + h2[i];
        if (tid == 0) col[rows] = nn;
    }
    cl.sync();  // no CTA leaves while another reads its shared memory
}

}  // namespace
}  // namespace tct

using namespace tct;

extern "C" int tct_arnoldi_step_fits(int64_t n, int rows) {
    return n >= 1 && n <= (int64_t)ARN_CTAS * ARN_SLICE && rows >= 1 && rows <= ARN_ROWS &&
           n * rows <= ARN_WORK;
}

extern "C" int tct_arnoldi_step(double* V, int64_t n, int rows, const double* w, double* col,
                                void* stream) {
    TCT_CHECK_ARG(tct_arnoldi_step_fits(n, rows),
                  "tct_arnoldi_step: %lld unknowns and %d basis vectors do not fit",
                  (long long)n, rows);
    TCT_CHECK_ARG(V && w && col, "tct_arnoldi_step: null pointer");
    if (cudaFuncSetAttribute(arnoldi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)ARN_SMEM) != cudaSuccess)
        return launch_status("tct_arnoldi_step shared memory");
    arnoldi_kernel<<<ARN_CTAS, ARN_THREADS, ARN_SMEM, as_stream(stream)>>>(V, n, rows, w, col);
    return launch_status("tct_arnoldi_step");
}
