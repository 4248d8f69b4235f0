// Sparse GAP kernel matrices for training, in FP64 (the reference's
// arithmetic):
//   K_NM energy rows    models/sparse_kernels.hh:104-131 (target Structure),
//                       :165-191 (target Atom);
//   K_NM gradient rows  models/sparse_kernels.hh:258-499 (with the negative
//                       stress rows of :405-425, :470-482);
//   K_MM                models/sparse_kernels.hh:141-156 with
//                       models/sparse_points.hh:144-170.
//
// All products run through the FP64 tile GEMM of dgemm.cuh. The gradient
// block needs (dX_i/dr_j . T_m) for every pair (i, j). With X = p / |p|,
//   dX/dr_j . T_m = (dp/dr_j . T_m - (x . dp/dr_j)(x . T_m)) / |p|,
// and dp/dr_j = dc/dr_j (x) c_i is nonzero only where one side has the
// neighbour's species: S n^2 (l+1) of the P n^2 (l+1) columns (a third at
// S = 5). So the pairs are listed by (species of i, species of j), the rows
// dp/dr_j / |p| of one such group are materialised in the short layout
// [l][b][n1][n2], and one GEMM per group contracts them with the sparse
// points of i's species rearranged for j's species. The epilogue subtracts
// the projection, scales by zeta (X_i . T_m)^(zeta-1) and adds the entry to
// row 3j + c and its negative to row 3i + c (the self pair's gradient is
// minus the sum of the others', image pairs of i left out,
// calculator_spherical_expansion.hh:2354-2358), and to the stress rows of
// the structure, so neither self-pair rows nor virial rows exist.
#include <cuda_runtime.h>

#include "common.cuh"
#include "dgemm.cuh"

namespace rgpu {
namespace {

// One warp per row of the sorted features; adds the planes of the dots.
__global__ void knm_rows_kernel(GapGroup g, const double * __restrict__ Km, int zeta,
                                const int32_t * __restrict__ center_of_row,
                                const int32_t * __restrict__ center_struct, int atom_target,
                                const int32_t * __restrict__ ucol, double * __restrict__ out, int64_t ldo) {
  const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (row >= g.row0[g.S]) return;
  int s = 0;
  while (row >= g.row0[s + 1]) ++s;
  const double * K = Km + g.koff[s] + (row - g.row0[s]) * g.ldk[s];
  const int64_t ci = center_of_row[row];
  double * o = out + (atom_target ? ci : int64_t(center_struct[ci])) * ldo;
  for (int m = threadIdx.x & 31; m < g.M[s]; m += 32) {
    double k = K[m];
    for (int p = 1; p < g.splits; ++p) k += K[p * g.plane + m];
    const double v = pow_zeta_d(k, zeta);
    if (atom_target)
      o[ucol[g.m0[s] + m]] = v;
    else
      atomicAdd(&o[ucol[g.m0[s] + m]], v);
  }
}

__global__ void dots_sum_kernel(int64_t n, int splits, int64_t plane, double * __restrict__ K) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double k = K[i];
  for (int p = 1; p < splits; ++p) k += K[p * plane + i];
  K[i] = k;
}

__global__ void kmm_scatter_kernel(int M, const double * __restrict__ K, int zeta,
                                   const int32_t * __restrict__ ucol, double * __restrict__ out,
                                   int64_t ldo) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= int64_t(M) * M) return;
  const int a = int(i / M), b = int(i - int64_t(a) * M);
  out[int64_t(ucol[a]) * ldo + ucol[b]] = pow_zeta_d(K[i], zeta);
}

constexpr int kMaxGroups = kMaxSpecies * kMaxSpecies;

// Pairs of the chunk by group g = species_i S + species_j (self pairs left
// out): their number, then their list. The order inside a group only moves
// the rounding of the atomic sums.
__global__ void __launch_bounds__(256)
pair_groups_kernel(ExpansionArgs a, int64_t p0, int64_t p1, const int32_t * __restrict__ pair_center, int S,
                   int32_t * __restrict__ cursor, int32_t * __restrict__ list) {
  __shared__ int32_t cnt[kMaxGroups], base[kMaxGroups];
  for (int g = threadIdx.x; g < S * S; g += blockDim.x) cnt[g] = 0;
  __syncthreads();
  const int64_t p = p0 + int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  int g = -1, rank = 0;
  if (p < p1) {
    const int32_t ci = pair_center[p];
    if (p != a.pair_off[ci]) {
      g = a.species_lut[a.types[a.center_atom[ci]]] * S + a.species_lut[a.types[a.pair_j[p]]];
      rank = atomicAdd(&cnt[g], 1);
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < S * S; k += blockDim.x)
    if (cnt[k]) base[k] = atomicAdd(&cursor[k], cnt[k]);
  __syncthreads();
  if (list && g >= 0) list[base[g] + rank] = int32_t(p);
}

__global__ void knm_points_kernel(FeatureDims fd, int M, int Kd, const double * __restrict__ T, int64_t ldt,
                                  double * __restrict__ Tq) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= int64_t(fd.S) * M * Kd) return;
  const int q = int(i % Kd), n = fd.n, L1 = fd.L + 1, nn = n * n;
  const int64_t sm = i / Kd;
  const int sj = int(sm / M);
  const double * t = T + (sm - int64_t(sj) * M) * ldt;
  const int l = q / (fd.S * nn), r = q - l * fd.S * nn;
  double v = 0.;
  if (l < L1) {
    const int b = r / nn, n1 = (r - b * nn) / n, n2 = r - b * nn - n1 * n;
    auto at = [&](int lo, int hi, int x, int y) {
      return t[((int64_t(lo * fd.S - lo * (lo - 1) / 2 + (hi - lo)) * n + x) * n + y) * L1 + l];
    };
    if (b == sj)
      v = at(b, b, n1, n2) + at(b, b, n2, n1);
    else if (sj < b)
      v = at(sj, b, n1, n2);
    else
      v = at(b, sj, n2, n1);
  }
  Tq[i] = v;
}

// One block per listed pair: the rows dp/dr_j[c] / |p| (c = x, y, z) in the
// short layout, and their products with x. dc/dr_j is formed once in shared
// memory (3 n K doubles); the rows are its contractions with c_i, four shared
// loads for three products, l slowest so that a warp's sums have one length
// and its stores are contiguous. Bound by those loads (47 k products per pair
// at S = 5, n = 8, l = 6) and by the 54 KB written.
__global__ void __launch_bounds__(128)
pair_rows_kernel(KnmGradArgs a, int Kd, const int32_t * __restrict__ list, const double * __restrict__ harmonics,
                 double * __restrict__ rows, double * __restrict__ proj) {
  extern __shared__ __align__(16) double sm[];
  const FeatureDims & fd = a.fd;
  const int n = fd.n, K = fd.K, W = fd.W, L1 = fd.L + 1, S = fd.S, Sn = fd.Sn, nn = n * n, nK = n * K;
  double * G = sm;              // [3][n][K]
  double * Cs = G + 3 * nK;     // [S n][K], after the three arrays of dc/dr below
  double * RI = Cs;             // [W] f_c / r RI
  double * P1 = RI + W;         // [W] dRI f_c + RI df_c
  double * Y = P1 + W;          // [4][K]
  __shared__ double red[3][4];
  const int64_t slot = blockIdx.x, p = list[slot];
  const int64_t ci = a.pair_center[p];
  const int sj = a.ea.species_lut[a.ea.types[a.ea.pair_j[p]]];
  const double r = a.ea.pair_dist[p];
  double fc, dfc;
  cutoff_fc_dfc(a.ea, r, fc, dfc);
  const SplinePos q = spline_pos(a.ea.sp, r);
  const double ca = q.a * q.a - 1., cb = q.b * q.b - 1., ea = 3. * q.a * q.a - 1., eb = 3. * q.b * q.b - 1.;
  const double * y0 = a.ea.sp.y + size_t(q.k) * W;
  const double * d0 = a.ea.sp.y2h + size_t(q.k) * W;
  for (int c = threadIdx.x; c < W; c += 128) {
    const double ya = __ldg(y0 + c), yb = __ldg(y0 + W + c), da = __ldg(d0 + c), db = __ldg(d0 + W + c);
    const double ri = q.a * (ya + ca * da) + q.b * (yb + cb * db);
    RI[c] = ri * fc / r;
    P1[c] = (yb - ya - ea * da + eb * db) / a.ea.sp.h * fc + ri * dfc;
  }
  for (int e = threadIdx.x; e < 4 * K; e += 128) Y[e] = harmonics[size_t(slot) * 4 * K + e];
  const double invn = a.inv_norm[ci];
  const double dir[3] = {a.ea.pair_dir[3 * p], a.ea.pair_dir[3 * p + 1], a.ea.pair_dir[3 * p + 2]};
  __syncthreads();
  const double * U = a.U + size_t(ci) * K * Sn + sj * n;
  double dot[3] = {0., 0., 0.};
  for (int e = threadIdx.x; e < nK; e += 128) {
    const int n1 = e / K, lm = e - n1 * K;
    int l = int(sqrtf(float(lm)));
    while (l * l > lm) --l;
    while ((l + 1) * (l + 1) <= lm) ++l;
    const double p1 = P1[n1 * L1 + l] * Y[lm] * invn, ri = RI[n1 * L1 + l] * invn;
    const double u = a.normalize ? U[lm * Sn + n1] : 0.;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double g = p1 * dir[c] + ri * Y[(c + 1) * K + lm];
      G[c * nK + e] = g;
      dot[c] = fma(u, g, dot[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    dot[c] = warp_sum(dot[c]);
    if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = dot[c];
  }
  __syncthreads();
  if (threadIdx.x < 3)
    proj[3 * slot + threadIdx.x] =
        red[threadIdx.x][0] + red[threadIdx.x][1] + red[threadIdx.x][2] + red[threadIdx.x][3];
  const double * Ci = a.C + size_t(ci) * Sn * K;
  for (int e = threadIdx.x; e < Sn * K; e += 128) Cs[e] = Ci[e];
  __syncthreads();
  double * out = rows + size_t(slot) * 3 * Kd;
  const int per_l = S * nn;
  for (int l = 0; l < L1; ++l) {
    const int M = 2 * l + 1;
    const double lf = 1. / sqrt(double(M)), lf2 = lf * 1.41421356237309504880168872420969808;
    for (int e = threadIdx.x; e < per_l; e += 128) {
      const int b = e / nn, n1 = (e - b * nn) / n, n2 = e - b * nn - n1 * n;
      const double * g = G + n1 * K + l * l;
      const double * c2 = Cs + (b * n + n2) * K + l * l;
      double s0 = 0., s1 = 0., s2 = 0.;
      for (int m = 0; m < M; ++m) {
        const double c = c2[m];
        s0 = fma(g[m], c, s0);
        s1 = fma(g[nK + m], c, s1);
        s2 = fma(g[2 * nK + m], c, s2);
      }
      const double f = b == sj ? lf : lf2;
      double * o = out + l * per_l + e;
      o[0] = s0 * f;
      o[Kd] = s1 * f;
      o[2 * Kd] = s2 * f;
    }
  }
  for (int e = L1 * per_l + threadIdx.x; e < Kd; e += 128) out[e] = out[Kd + e] = out[2 * Kd + e] = 0.;
}

// Entry (3 k + c, m) of a group's product: row c of pair list[k] against
// sparse point m of the group's central species.
struct PairEntries {
  struct Row {
    const double * k;  // x . T of the centre
    double proj, ra, rb;
    double * oj;
    double * oi;  // null for an image of the centre
    double * sa;  // stress rows, or null
    double * sb;
  };
  const int32_t * list;
  const double * proj;
  const int32_t * pair_center;
  const int32_t * pair_j;
  const int32_t * center_atom;
  const int32_t * row_of_center;
  const int32_t * center_struct;
  const double * pair_dist;
  const double * pair_dir;
  const double * K;  // of the species, rows from row0
  int64_t row0, ldk;
  int zeta;
  const int32_t * ucol;
  double * out;
  int64_t ldo, stress_row0;
  __device__ __forceinline__ Row row(int64_t r) const {
    const int64_t k = r / 3;
    const int c = int(r - 3 * k);
    const int64_t p = list[k], ci = pair_center[p];
    const int32_t j = pair_j[p], i = center_atom[ci];
    Row w;
    w.k = K + (int64_t(row_of_center[ci]) - row0) * ldk;
    w.proj = proj[r];
    w.oj = out + (3 * int64_t(j) + c) * ldo;
    w.oi = j == i ? nullptr : out + (3 * int64_t(i) + c) * ldo;
    w.sa = w.sb = nullptr;
    w.ra = w.rb = 0.;
    if (stress_row0 >= 0) {
      // r_ji (x) d/dr_j: xx and xz from x, yy and xy from y, zz and yz from z
      // (models/sparse_kernels.hh:405-425)
      const int pair[3] = {2, 0, 1}, row_b[3] = {4, 5, 3};
      const double dist = -pair_dist[p];
      double * s = out + (stress_row0 + 6 * int64_t(center_struct[ci])) * ldo;
      w.sa = s + c * ldo;
      w.ra = dist * pair_dir[3 * p + c];
      w.sb = s + row_b[c] * ldo;
      w.rb = dist * pair_dir[3 * p + pair[c]];
    }
    return w;
  }
  __device__ __forceinline__ void put(const Row & w, int m, double v, int) const {
    const double k = w.k[m];
    // zeta k^(zeta-1), exactly 1 for zeta = 1 (models/sparse_kernels.hh:320-331)
    const double x = (v - w.proj * k) * (zeta > 1 ? double(zeta) * pow_zeta_d(k, zeta - 1) : 1.);
    const int col = ucol[m];
    atomicAdd(w.oj + col, x);
    if (w.oi) atomicAdd(w.oi + col, -x);
    if (w.sa) {
      atomicAdd(w.sa + col, w.ra * x);
      atomicAdd(w.sb + col, w.rb * x);
    }
  }
};

}  // namespace

void launch_knm_rows(const GapGroup & g, const double * K, int zeta, const int32_t * center_of_row,
                     const int32_t * center_struct, bool atom_target, const int32_t * ucol, double * out, int64_t ldo,
                     cudaStream_t st) {
  if (g.row0[g.S] <= 0) return;
  knm_rows_kernel<<<div_up(g.row0[g.S] * 32, 256), 256, 0, st>>>(g, K, zeta, center_of_row, center_struct,
                                                                int(atom_target), ucol, out, ldo);
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

void launch_dots_sum(const GapGroup & g, double * K, cudaStream_t st) {
  if (g.plane <= 0 || g.splits < 2) return;
  dots_sum_kernel<<<div_up(g.plane, 256), 256, 0, st>>>(g.plane, g.splits, g.plane, K);
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

void launch_kmm_scatter(int M, const double * K, int zeta, const int32_t * ucol, double * out, int64_t ldo,
                        cudaStream_t st) {
  if (M <= 0) return;
  kmm_scatter_kernel<<<div_up(int64_t(M) * M, 256), 256, 0, st>>>(M, K, zeta, ucol, out, ldo);
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

void launch_knm_points(const FeatureDims & fd, int M, const double * T, int64_t ldt, double * Tq, cudaStream_t st) {
  const int Kd = knm_row_len(fd);
  const int64_t n = int64_t(fd.S) * M * Kd;
  if (n <= 0) return;
  knm_points_kernel<<<unsigned((n + 255) / 256), 256, 0, st>>>(fd, M, Kd, T, ldt, Tq);
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

size_t knm_pair_bytes(const FeatureDims & fd) {
  return sizeof(double) * (3 * size_t(knm_row_len(fd)) + 3 + 4 * size_t(fd.K)) + sizeof(int32_t);
}

void launch_knm_gradient(const KnmGradArgs & a, DevBuf & list_buf, DevBuf & scratch, cudaStream_t st) {
  const FeatureDims & fd = a.fd;
  const int S = fd.S, Kd = knm_row_len(fd);
  const int64_t np = a.p1 - a.p0;
  if (np <= 0) return;
  // group sizes, then the list
  list_buf.ensure(sizeof(int32_t) * (size_t(np) + 2 * kMaxGroups));
  int32_t * cursor = list_buf.as<int32_t>();
  int32_t * list = cursor + kMaxGroups;
  RGPU_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int32_t) * S * S, st));
  const unsigned blocks = unsigned((np + 255) / 256);
  pair_groups_kernel<<<blocks, 256, 0, st>>>(a.ea, a.p0, a.p1, a.pair_center, S, cursor, nullptr);
  RGPU_LAUNCHED();
  int32_t count[kMaxGroups], start[kMaxGroups + 1];
  RGPU_CUDA(cudaMemcpyAsync(count, cursor, sizeof(int32_t) * S * S, cudaMemcpyDeviceToHost, st));
  RGPU_CUDA(cudaStreamSynchronize(st));
  start[0] = 0;
  for (int g = 0; g < S * S; ++g) start[g + 1] = start[g] + count[g];
  const int64_t n_list = start[S * S];
  if (n_list == 0) return;
  RGPU_CUDA(cudaMemcpyAsync(cursor, start, sizeof(int32_t) * S * S, cudaMemcpyHostToDevice, st));
  pair_groups_kernel<<<blocks, 256, 0, st>>>(a.ea, a.p0, a.p1, a.pair_center, S, cursor, list);
  RGPU_LAUNCHED();
  scratch.ensure(sizeof(double) * size_t(n_list) * (3 * size_t(Kd) + 4 + 4 * size_t(fd.K)) + 256);
  double * rows = scratch.as<double>();
  double * harmonics = rows + size_t(n_list) * 3 * Kd;
  double * proj = harmonics + size_t(n_list) * 4 * fd.K;
  launch_pair_harmonics_fp64(a.ea, n_list, list, harmonics, st);
  const size_t smem =
      sizeof(double) * (3 * size_t(fd.nK) + std::max(size_t(fd.Sn) * fd.K, 2 * size_t(fd.W) + 4 * size_t(fd.K)));
  RGPU_CUDA(cudaFuncSetAttribute(pair_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  pair_rows_kernel<<<unsigned(n_list), 128, smem, st>>>(a, Kd, list, harmonics, rows, proj);
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
  DgGroup<PairEntries> d{};
  d.splits = 1;
  for (int g = 0; g < S * S; ++g) {
    const int si = g / S, sj = g - si * S;
    if (count[g] > 0 && a.dots->M[si] > 0) {
      PairEntries e{list + start[g],
                    proj + 3 * size_t(start[g]),
                    a.pair_center,
                    a.ea.pair_j,
                    a.ea.center_atom,
                    a.row_of_center,
                    a.center_struct,
                    a.ea.pair_dist,
                    a.ea.pair_dir,
                    a.K + a.dots->koff[si],
                    a.dots->row0[si],
                    a.dots->ldk[si],
                    a.zeta,
                    a.ucol + a.dots->m0[si],
                    a.out,
                    a.ldo,
                    a.stress_row0};
      d.p[d.n++] = {3 * int64_t(count[g]), a.dots->M[si], Kd, rows + size_t(start[g]) * 3 * Kd, Kd,
                    a.Tq + (size_t(sj) * a.M + a.dots->m0[si]) * Kd, Kd, e};
    }
    if (d.n == kDgMaxProblems || (g + 1 == S * S && d.n > 0)) {
      launch_dgemm<true>(d, true, st);
      d.n = 0;
    }
  }
}

}  // namespace rgpu
