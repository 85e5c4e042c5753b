// mrmg_dist.cu -- configuration distances and costs
// (problems/core/configuration.py): batch_config_dist / NpConfiguration._batch_dist
// (:303-349), compute_sliced_euclidean_dists (:101-126), the sum / max /
// max+w*sum / abs-max reductions (:129-219) and batch_config_cost (:437-510).
//
// Every value is the FP64 result of the reference's own operation sequence
// (sequential sums of d*d without fusion, IEEE sqrt, strict '>' maxima), so
// outputs are bit-identical to the reference.  These kernels are bound by the
// FP64 pipe on GB300 (1.7 lane operations per clock and SM), not by HBM: squares,
// roots and maxima therefore run on the integer pipes (mrmg_exact.cuh), two FP64
// operations per coordinate are left.  1,000 x 10,000 distances: euclidean in 4
// coordinates 394 -> 145 us (the 7 FP64 operations alone 142 us; all 19 were 390),
// in 28 1,850 -> 1,125 us, max over agents 2,400 -> 1,060 us, max 1,700 -> 585 us.
#include "mrmg_internal.cuh"

namespace mrmg {

namespace {

constexpr int kQTile = 16;        // queries per CTA (shared memory)
constexpr int kMaxTileD = 128;    // coordinates staged per query
constexpr int kNodesPerCta = 128;
constexpr int kMinStaged = 4;     // queries from which staging a CTA's nodes pays (one query, 12,000 nodes, 28 coordinates:
                                  // 37 us in place, 42 us staged)
// Distances of nodes read in place, too few to keep the FP64 pipe busy: the FP64
// instructions, whose loads and chains overlap across coordinates (97 coordinates, 17
// queries: 3,000 nodes 213 us, integer squares 498 us; 15,000 nodes 222 and 499 us);
// 60 queries on 15,000 nodes 727 us in FP64 instructions, 552 us.
constexpr long long kFewDists = 1ll << 18;
constexpr size_t kMaxNodeTile = 96 * 1024;   // bytes of staged nodes: two CTAs per SM at least

// out[q, m] = dist(queries[q] - nodes[m]).  A node per thread, the tile's
// queries one after another.  DM > 0: euclidean in end_all <= DM coordinates, the
// node's held in registers.  Else the CTA's nodes are staged in shared memory by
// coordinate (XS; read from global memory, a row per lane, the L1 cache bound 28
// coordinates at 0.94 ms per 1,000 x 10,000), or read in place where they do not fit.
template <int DM, bool XS, bool FAST1 = false>
__global__ void __launch_bounds__(kNodesPerCta) dist_matrix_kernel(const double* __restrict__ qs, long long Q,
                                                                   const double* __restrict__ nodes, long long M,
                                                                   SliceTab t, int metric, double* __restrict__ out) {
  extern __shared__ double sq[];   // queries [kQTile][D] (up to kMaxTileD coordinates), then XS: nodes [D][kNodesPerCta]
  const int D = t.D;
  double* xs = sq + kQTile * D;
  const long long q0 = (long long)blockIdx.y * kQTile;
  const int nq = (int)min((long long)kQTile, Q - q0);
  const bool staged = D <= kMaxTileD;
  if (staged)
    for (int i = threadIdx.x; i < nq * D; i += kNodesPerCta) sq[i] = qs[q0 * D + i];
  __syncthreads();
  for (long long m0 = blockIdx.x * (long long)kNodesPerCta; m0 < M; m0 += (long long)gridDim.x * kNodesPerCta) {
    const long long m = m0 + threadIdx.x;
    const double* x = nodes + m * D;
    if constexpr (XS) {
      const int n = (int)min((long long)kNodesPerCta, M - m0) * D;
      for (int i = threadIdx.x; i < n; i += kNodesPerCta) xs[(i % D) * kNodesPerCta + i / D] = nodes[m0 * D + i];
      __syncthreads();
    }
    if (m < M) {
      double xr[DM > 0 ? DM : 1];
      if constexpr (DM > 0) {
#pragma unroll
        for (int k = 0; k < DM; k++) xr[k] = k < t.end_all ? x[k] : 0.0;
      }
      for (int j = 0; j < nq; j++) {
        const double* qq = staged ? sq + j * D : qs + (q0 + j) * D;
        double v;
        if constexpr (DM > 0) {
          v = square_rn(__dsub_rn(qq[0], xr[0]));
#pragma unroll
          for (int k = 1; k < DM; k++)
            if (k < t.end_all) v = __dadd_rn(v, square_rn(__dsub_rn(qq[k], xr[k])));
          v = sqrt_rn(v);
        } else {
          v = dist_of<FAST1>(t, metric, [&](int k) { return __dsub_rn(qq[k], XS ? xs[k * kNodesPerCta + threadIdx.x] : x[k]); });
        }
        out[(q0 + j) * M + m] = v;
      }
    }
    if constexpr (XS) __syncthreads();   // the next nodes overwrite these
  }
}

// _batch_config_cost_impl on diff rows; mode 0: starts[0] - ends[m],
// 1: starts[m] - ends[m], 2: starts[m+1] - starts[m] (path form)
__global__ void cost_kernel(const double* __restrict__ a, const double* __restrict__ b, long long M, SliceTab t,
                            int cmetric, int red, double w, int mode, double* __restrict__ out) {
  const int D = t.D;
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < M; m += (long long)gridDim.x * blockDim.x) {
    const double* x;
    const double* y;
    if (mode == 0) { x = a; y = b + m * D; }
    else if (mode == 1) { x = a + m * D; y = b + m * D; }
    else { x = a + (m + 1) * D; y = a + m * D; }
    double mx = 0.0, sm = 0.0;
    for (int i = 0; i < t.A; i++) {
      double v;
      if (cmetric == MRMG_COST_EUCLIDEAN) {
        v = sqrt_rn(square_sum(t.s[i], t.e[i], [&](int k) { return __dsub_rn(x[k], y[k]); }));
      } else {
        // np.max(np.abs(diff[:, s:e])): exact; a NaN anywhere propagates
        v = fabs(__dsub_rn(x[t.s[i]], y[t.s[i]]));
        for (int k = t.s[i] + 1; k < t.e[i]; k++) { double d = fabs(__dsub_rn(x[k], y[k])); if (d > v || d != d) v = d; }
      }
      if (red == MRMG_REDUCE_MAX) {              // compute_max_sum_reduction (:150-171)
        if (i == 0) { mx = v; sm = v; }
        else { if (v > mx) mx = v; sm = __dadd_rn(sm, v); }
      } else {                                   // compute_sum_reduction (:129-147)
        sm = __dadd_rn(sm, v);
      }
    }
    out[m] = red == MRMG_REDUCE_MAX ? __dadd_rn(mx, __dmul_rn(w, sm)) : sm;
  }
}

int grid_for(long long n, int threads, int cap) {
  long long g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  return (int)(g < cap ? g : cap);
}

}  // namespace

cudaError_t dist_matrix(const double* qs, long long Q, const double* nodes, long long M, const SliceTab& t, int metric,
                        double* out, int num_sms, cudaStream_t st) {
  if (Q == 0 || M == 0) return cudaSuccess;
  long long qtiles = (Q + kQTile - 1) / kQTile;
  if (qtiles > 65535) return cudaErrorInvalidValue;
  const dim3 grid(grid_for(M, kNodesPerCta, num_sms * 16), (unsigned)qtiles);
  const bool eu = metric == MRMG_METRIC_EUCLIDEAN && t.end_all >= 1 && t.D <= kMaxTileD;
  const size_t tile = sizeof(double) * kNodesPerCta * t.D, qt = t.D <= kMaxTileD ? sizeof(double) * kQTile * t.D : 0;
  cudaError_t e = cudaSuccess;
  if (eu && t.end_all <= 4) {
    dist_matrix_kernel<4, false><<<grid, kNodesPerCta, qt, st>>>(qs, Q, nodes, M, t, metric, out);
  } else if (eu && t.end_all <= 8) {
    dist_matrix_kernel<8, false><<<grid, kNodesPerCta, qt, st>>>(qs, Q, nodes, M, t, metric, out);
  } else if (tile <= kMaxNodeTile && Q >= kMinStaged) {
    e = allow_max_smem(dist_matrix_kernel<0, true>);
    if (e == cudaSuccess)
      dist_matrix_kernel<0, true><<<grid, kNodesPerCta, qt + tile, st>>>(qs, Q, nodes, M, t, metric, out);
  } else if (Q * M < kFewDists) {
    dist_matrix_kernel<0, false, true><<<grid, kNodesPerCta, qt, st>>>(qs, Q, nodes, M, t, metric, out);
  } else {
    dist_matrix_kernel<0, false><<<grid, kNodesPerCta, qt, st>>>(qs, Q, nodes, M, t, metric, out);
  }
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t batch_cost(const double* a, const double* b, long long M, const SliceTab& t, int cmetric, int red, double w,
                       int mode, double* out, int num_sms, cudaStream_t st) {
  if (M <= 0) return cudaSuccess;
  cost_kernel<<<grid_for(M, 256, num_sms * 16), 256, 0, st>>>(a, b, M, t, cmetric, red, w, mode, out);
  return cudaGetLastError();
}

}  // namespace mrmg
