// Dense contractions of the GAP model.
//
// Forward, per central species s:  k = X_s T_s^T,  e_i = sum_m alpha_m k^zeta,
// W = alpha zeta k^(zeta-1)   (models/sparse_kernels.hh:104-131,
// models/sparse_kernel_predict.hh:130-145, models/kernels.hh:48-61).
// Backward: dE/dX_s = W T_s (the "sparse_point_scaled" contraction of
// models/sparse_kernel_predict.hh:141-143, done for all centres at once).
//
// In FP64 here, on the tensor-core tiles of dgemm.cuh; the FP32 path's, with
// the pointwise part in the forward's epilogue, are in gemm_tc.cu.
#include <cuda_runtime.h>

#include "common.cuh"
#include "dgemm.cuh"

namespace rgpu {
namespace {

// One warp per row of the sorted features; adds the planes of the dots.
__global__ void gap_pointwise_fp64_kernel(GapGroup g, double * __restrict__ Km, const double * __restrict__ alpha,
                                          int zeta, double * __restrict__ e_row) {
  const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= g.row0[g.S]) return;
  int s = 0;
  while (row >= g.row0[s + 1]) ++s;
  double * K = Km + g.koff[s] + (row - g.row0[s]) * g.ldk[s];
  double e = 0.;
  for (int m = lane; m < g.M[s]; m += 32) {
    double k = K[m];
    for (int p = 1; p < g.splits; ++p) k += K[p * g.plane + m];
    const double al = alpha[g.m0[s] + m];
    e += al * pow_zeta_d(k, zeta);
    K[m] = al * (zeta * pow_zeta_d(k, zeta - 1));
  }
  e = warp_sum(e);
  if (lane == 0) e_row[row] = e;
}

__global__ void energy_reduce_kernel(int64_t rows, EnergyParts parts, const float * __restrict__ e_part,
                                     const double * __restrict__ e_row, const int32_t * __restrict__ center_of_row,
                                     const int32_t * __restrict__ center_struct,
                                     double * __restrict__ E) {
  const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  double e = 0.;
  int key = -1;
  if (r < rows) {
    if (e_row) {
      e = e_row[r];
    } else {
      int s = 0;
      while (r >= parts.row0[s + 1]) ++s;
      const int64_t ld = parts.row0[s + 1] - parts.row0[s];
      const float * p = e_part + parts.ofs[s] + (r - parts.row0[s]);
      for (int t = 0; t < parts.parts[s]; ++t) e += double(p[int64_t(t) * ld]);
    }
    key = center_struct[center_of_row[r]];
  }
  // the warp's rows of one structure are summed first, so a structure with
  // many centres (one large box) takes one atomic per warp, not per row
  const int lane = threadIdx.x & 31;
  double sum = 0.;
  int leader = 32;
#pragma unroll 4
  for (int src = 0; src < 32; ++src) {
    const double v = __shfl_sync(0xffffffffu, e, src);
    const int k = __shfl_sync(0xffffffffu, key, src);
    if (k == key) {
      sum += v;
      leader = min(leader, src);
    }
  }
  if (key >= 0 && leader == lane) atomicAdd(&E[key], sum);
}

}  // namespace

void gemm_nt_fp64(int64_t M, int64_t N, int64_t K, const double * A, int64_t lda, const double * B,
                  int64_t ldb, double * C, int64_t ldc, cudaStream_t st) {
  DgGroup<DgStoreC> g{};
  g.n = g.splits = 1;
  g.p[0] = {M, int(N), int(K), A, lda, B, ldb, DgStoreC{C, ldc, 0}};
  launch_dgemm<true>(g, dgemm_aligned(A, lda) && dgemm_aligned(B, ldb), st);
}

void gap_dots_split(GapGroup & g, int K) {
  int64_t tiles = 0;
  for (int s = 0; s < g.S; ++s)
    if (g.M[s] > 0) tiles += dgemm_tiles(g.rows[s], g.M[s]);
  g.splits = dgemm_splits(tiles, K);
}

void launch_gap_dots_fp64(const GapGroup & g, int K, const double * X, int64_t ldx, const double * T, int64_t ldt,
                          double * Kmat, cudaStream_t st) {
  DgGroup<DgStoreC> d{};
  d.splits = g.splits;
  for (int s = 0; s < g.S; ++s)
    if (g.rows[s] > 0 && g.M[s] > 0)
      d.p[d.n++] = {g.rows[s], g.M[s], K, X + g.row0[s] * ldx, ldx, T + g.m0[s] * ldt, ldt,
                    DgStoreC{Kmat + g.koff[s], g.ldk[s], g.plane}};
  launch_dgemm<true>(d, dgemm_aligned(X, ldx) && dgemm_aligned(T, ldt), st);
}

void launch_gap_scaled_fp64(const GapGroup & g, int D, const double * W, const double * T, int64_t ldt, double * t,
                            int64_t ld, cudaStream_t st) {
  DgGroup<DgStoreC> d{};
  d.splits = 1;
  bool aligned = dgemm_aligned(W, 0) && dgemm_aligned(T, ldt);
  for (int s = 0; s < g.S; ++s)
    if (g.rows[s] > 0 && g.M[s] > 0) {
      aligned = aligned && (g.koff[s] & 1) == 0;
      d.p[d.n++] = {g.rows[s], D, g.M[s], W + g.koff[s], g.ldk[s], T + g.m0[s] * ldt, ldt,
                    DgStoreC{t + g.row0[s] * ld, ld, 0}};
    }
  launch_dgemm<false>(d, aligned, st);
}

void launch_gap_pointwise_fp64(const GapGroup & g, double * Kmat, const double * alpha, int zeta, double * e_row,
                               cudaStream_t st) {
  if (g.row0[g.S] <= 0) return;
  gap_pointwise_fp64_kernel<<<div_up(g.row0[g.S] * 32, 256), 256, 0, st>>>(g, Kmat, alpha, zeta, e_row);
  RGPU_LAUNCHED();
}

void launch_energy_reduce(int64_t rows, const EnergyParts & parts, const float * e_part, const double * e_row_fp64,
                          const int32_t * center_of_row, const int32_t * center_struct, double * energies,
                          cudaStream_t st) {
  if (rows <= 0) return;
  energy_reduce_kernel<<<div_up(rows, 256), 256, 0, st>>>(rows, parts, e_part, e_row_fp64, center_of_row,
                                                         center_struct, energies);
  RGPU_LAUNCHED();
}

}  // namespace rgpu
