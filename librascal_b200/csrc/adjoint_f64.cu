// FP64 adjoint of the GAP energy: dE/dx -> dE/dc per centre, then the forces
// (and the negative stress) from one pass over the pairs that recomputes
// dc/dr, as the FP32 path does (ps_fast.cu, adjoint.cu), in the reference's
// precision and its dense feature order.
//
// The reference contracts the materialised dX/dr of every pair with the
// scaled sparse points t_i = sum_m w_m T_m (models/sparse_kernel_predict.hh:
// 130-172). The same sums in another order need no pair gradient: t_i goes
// back through the normalisation and the power spectrum once per centre, and
// only dE/dc_i (S n (l+1)^2 values) meets the pairs. A pair costs about
// 4 n (l+1)^2 multiplications instead of 6 D: at S = 5, n = 8, l = 6 that is
// 1.6 k instead of 40 k, and 3 D doubles per pair (161 KB) are neither
// written nor read back.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace rgpu {
namespace {

constexpr int kBwdThreads = 256;
constexpr int kPairThreads = 64;
constexpr int kNV = 8;  // radial channels staged in registers at a time
constexpr double kSqrt2 = 1.41421356237309504880168872420969808;

// Distance between the l planes of the shared gradient: P n^2 rounded up to
// 5 modulo 16 doubles, so that the row's values, which arrive with l
// fastest, fall in different banks.
__host__ __device__ inline int l_plane(int pnn) { return pnn + ((5 - pnn) & 15); }

// Per centre: G = (t - x (x.t)) / |p| for the dense row (t = dE/dx), kept in
// shared memory as [l][key][n1][n2], then
//   dE/dc_(a n1 l m) = lf_l sum_b s_ab sum_n2 G~_ab(n1 n2 l) c_(b n2 l m),
// s_ab = sqrt2 for a != b (calculator_spherical_invariants.hh:747-794), with
// G~_ab = G_(ab)(n1 n2) for a < b, G_(ba)(n2 n1) for a > b and their sum for
// a = b. One block per centre; a task is two rows n1 and four values m of one
// l, so two loads of G and four of c feed eight products. Bound by the two
// passes over x and t (2 x 54 KB per centre at S = 5, n = 8, l = 6); the
// contraction is 78 k FMAs, a fifth of that time.
template <int L>
__global__ void __launch_bounds__(kBwdThreads)
ps_bwd_f64_kernel(PsArgs a, int plane, const double * __restrict__ C, const double * __restrict__ X,
                  const double * __restrict__ inv_norm, const double * __restrict__ t, double * __restrict__ dC) {
  constexpr int L1 = L + 1, K = L1 * L1;
  extern __shared__ __align__(16) double smd[];
  const FeatureDims fd = a.fd;
  const int S = fd.S, n = fd.n, Sn = fd.Sn, nn2 = n * n;
  double * Cs = smd;             // [S n][K]
  double * Gs = smd + Sn * K;    // [L1][plane]
  __shared__ double red[kBwdThreads / 32];
  const int64_t ci = blockIdx.x;
  const double * Ci = C + size_t(ci) * Sn * K;
  for (int e = threadIdx.x; e < Sn * K; e += kBwdThreads) Cs[e] = Ci[e];
  const size_t row = size_t(a.row_of_center[ci]) * fd.Dpad;
  const double * xr = X + row;
  const double * tr = t + row;
  const double invn = inv_norm[ci];
  double dot = 0.;
  for (int d = threadIdx.x; d < fd.D; d += kBwdThreads) {
    const double v = tr[d];
    if (a.normalize) dot = fma(v, xr[d], dot);
    Gs[(d % L1) * plane + d / L1] = v;  // d / L1 = key n^2 + n1 n + n2
  }
  if (a.normalize) {
    dot = warp_sum(dot);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
    __syncthreads();
    dot = 0.;
#pragma unroll
    for (int w = 0; w < kBwdThreads / 32; ++w) dot += red[w];
    for (int d = threadIdx.x; d < fd.D; d += kBwdThreads) {
      double * g = Gs + (d % L1) * plane + d / L1;
      *g = (*g - xr[d] * dot) * invn;
    }
  }
  __syncthreads();
  const uint32_t pm = a.present[ci];
  constexpr int kChunks = offp(L1) / 4;  // chunks of four m, l by l
  const int n_pairs = (n + 1) >> 1;
  for (int task = threadIdx.x; task < S * n_pairs * kChunks; task += kBwdThreads) {
    const int rows = task / kChunks, ch = task - rows * kChunks;
    const int sa = rows / n_pairs, n1 = 2 * (rows - sa * n_pairs);
    if (!((pm >> sa) & 1u)) continue;  // no pair of the species: its dE/dc is never read
    int l = 0;
#pragma unroll
    for (int q = 1; q <= L; ++q) l += (4 * ch >= offp(q));
    const int m0 = 4 * ch - offp_rt(l), M = 2 * l + 1;
    const bool two = n1 + 1 < n;
    const double * Gl = Gs + l * plane;
    double acc0[4] = {0., 0., 0., 0.}, acc1[4] = {0., 0., 0., 0.};
    for (int sb = 0; sb < S; ++sb) {
      if (!((pm >> sb) & 1u)) continue;
      const int lo = min(sa, sb), hi = max(sa, sb);
      const double * G = Gl + (lo * S - lo * (lo - 1) / 2 + (hi - lo)) * nn2;
      const double * c = Cs + sb * n * K + l * l + m0;
      double p0[4] = {0., 0., 0., 0.}, p1[4] = {0., 0., 0., 0.};
      // the key as stored (n1 indexes its rows) and transposed
#pragma unroll
      for (int form = 0; form < 2; ++form) {
        if (form == 0 ? sa > sb : sa < sb) continue;
        const double * g = form == 0 ? G + n1 * n : G + n1;
        const int next_row = two ? (form == 0 ? n : 1) : 0, next_col = form == 0 ? 1 : n;
        for (int n2 = 0; n2 < n; ++n2) {
          const double g0 = g[n2 * next_col], g1 = g[n2 * next_col + next_row];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (m0 + e < M) {
              const double v = c[n2 * K + e];
              p0[e] = fma(g0, v, p0[e]);
              p1[e] = fma(g1, v, p1[e]);
            }
        }
      }
      const double s = sa == sb ? 1. : kSqrt2;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc0[e] = fma(s, p0[e], acc0[e]);
        acc1[e] = fma(s, p1[e], acc1[e]);
      }
    }
    const double lf = 1. / sqrt(double(M));
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (m0 + e < M) {
        double * o = dC + (size_t(ci) * K + (l * l + m0 + e)) * Sn + sa * n + n1;
        o[0] = acc0[e] * lf;
        if (two) o[1] = acc1[e] * lf;
      }
  }
}

// One thread per pair, as adjoint.cu: per l the radial values RI and
// p1 = dRI f_c + RI df_c of up to kNV channels are staged in registers and
// the spherical-harmonics recurrence streams (Y, grad Y) past them; larger n
// takes several passes. Bound by the latency of one pair's chain (about
// 1 500 dependent FP64 operations at l = 6), so the blocks are small: 64
// threads spread even a few thousand pairs over the chip.
template <int L>
__global__ void __launch_bounds__(kPairThreads)
pair_adjoint_f64_kernel(ExpansionArgs a, const int32_t * __restrict__ pair_center, int64_t n_pairs,
                        const double * __restrict__ dC, double * __restrict__ F,
                        const int32_t * __restrict__ center_struct, double * __restrict__ stress) {
  constexpr int L1 = L + 1, K = L1 * L1;
  const int W = a.fd.W, n = a.fd.n, Sn = a.fd.Sn;
  const int lane = threadIdx.x & 31;
  {
    // the list's own total bounds the loop (below n_pairs when the list was
    // built to a capacity)
    const int64_t listed = a.pair_off[a.n_centers];
    if (listed < n_pairs) n_pairs = listed;
  }
  const int64_t p = int64_t(blockIdx.x) * kPairThreads + threadIdx.x;
  if (p - lane >= n_pairs) return;  // whole warps: the sums below shuffle across lanes
  const int32_t ci = p < n_pairs ? pair_center[p] : -1;
  double g[3] = {0., 0., 0.}, t6[6] = {0., 0., 0., 0., 0., 0.};
  int32_t j = -1, self_atom = -1;
  // the self pair carries no force of its own: the other pairs' F_i terms do
  if (ci >= 0 && p != a.pair_off[ci]) {
    self_atom = a.center_atom[ci];
    const double r = a.pair_dist[p];
    j = a.pair_j[p];
    const int s = a.species_lut[a.types[j]];
    double fc, dfc;
    cutoff_fc_dfc(a, r, fc, dfc);
    const SplinePos q = spline_pos(a.sp, r);
    const double ca = q.a * q.a - 1., cb = q.b * q.b - 1., ea = 3. * q.a * q.a - 1., eb = 3. * q.b * q.b - 1.;
    const double * y0 = a.sp.y + size_t(q.k) * W;
    const double * d0 = a.sp.y2h + size_t(q.k) * W;
    const double dx = a.pair_dir[3 * p], dy = a.pair_dir[3 * p + 1], dz = a.pair_dir[3 * p + 2];
    const double * E0 = dC + size_t(ci) * K * Sn + s * n;
    double sY = 0., sx = 0., sy = 0., sz = 0.;
    for (int c0 = 0; c0 < n; c0 += kNV) {
      double rl[kNV], pl[kNV];
      const double * E = E0 + c0;
      spherical_harmonics<L, true, double>(
          dx, dy, dz,
          [&](int lm, double y, double gx, double gy, double gz) {
            double A = 0., B = 0.;
            const double * e = E + lm * Sn;
#pragma unroll
            for (int k = 0; k < kNV; ++k)
              if (c0 + k < n) {
                const double ev = __ldg(e + k);
                A = fma(ev, pl[k], A);
                B = fma(ev, rl[k], B);
              }
            sY = fma(A, y, sY);
            sx = fma(B, gx, sx);
            sy = fma(B, gy, sy);
            sz = fma(B, gz, sz);
          },
          [&](int l) {
#pragma unroll
            for (int k = 0; k < kNV; ++k)
              if (c0 + k < n) {
                const int c = (c0 + k) * L1 + l;
                const double ya = __ldg(y0 + c), yb = __ldg(y0 + W + c), da = __ldg(d0 + c), db = __ldg(d0 + W + c);
                const double ri = q.a * (ya + ca * da) + q.b * (yb + cb * db);
                const double dri = (yb - ya - ea * da + eb * db) / a.sp.h;
                rl[k] = ri;
                pl[k] = dri * fc + ri * dfc;
              }
          });
    }
    const double fr = fc / r;
    g[0] = dx * sY + fr * sx;
    g[1] = dy * sY + fr * sy;
    g[2] = dz * sY + fr * sz;
    if (stress) {
      // r_ji (x) g_ij, Voigt xx yy zz yz xz xy (sparse_kernel_predict.hh:355-366)
      const double rx = -r * dx, ry = -r * dy, rz = -r * dz;
      t6[0] = rx * g[0];
      t6[1] = ry * g[1];
      t6[2] = rz * g[2];
      t6[3] = ry * g[2];
      t6[4] = rz * g[0];
      t6[5] = rx * g[1];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) atomicAdd(&F[3 * size_t(j) + k], -g[k]);
  }
  // F_i += g unless j is a periodic image of i (calculator_spherical_expansion.hh:
  // 2354-2358): the centre's pairs are consecutive lanes, so a segmented warp
  // scan leaves each run's sum in its last lane
  if (j < 0 || j == self_atom) g[0] = g[1] = g[2] = 0.;
  const int32_t sid = (stress && ci >= 0) ? center_struct[ci] : -1;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t cu = __shfl_up_sync(0xffffffffu, ci, off);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double u = __shfl_up_sync(0xffffffffu, g[k], off);
      if (lane >= off && cu == ci) g[k] += u;
    }
    if (stress) {
      const int32_t su = __shfl_up_sync(0xffffffffu, sid, off);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double u = __shfl_up_sync(0xffffffffu, t6[k], off);
        if (lane >= off && su == sid) t6[k] += u;
      }
    }
  }
  const int32_t cn = __shfl_down_sync(0xffffffffu, ci, 1), sn = __shfl_down_sync(0xffffffffu, sid, 1);
  if (ci >= 0 && (lane == 31 || cn != ci)) {
    const int32_t ia = a.center_atom[ci];
#pragma unroll
    for (int k = 0; k < 3; ++k) atomicAdd(&F[3 * size_t(ia) + k], g[k]);
  }
  if (sid >= 0 && (lane == 31 || sn != sid))
#pragma unroll
    for (int k = 0; k < 6; ++k) atomicAdd(&stress[6 * size_t(sid) + k], t6[k]);
}

// Spherical harmonics and their gradients of pairs list[0..n) (pair indices
// of the neighbour list), for the training matrices: out[k] = [4][K], the
// values and their x, y, z derivatives.
template <int L>
__global__ void __launch_bounds__(kPairThreads)
pair_harmonics_kernel(ExpansionArgs a, int64_t n, const int32_t * __restrict__ list, double * __restrict__ out) {
  constexpr int K = (L + 1) * (L + 1);
  const int64_t k = int64_t(blockIdx.x) * kPairThreads + threadIdx.x;
  if (k >= n) return;
  const int64_t p = list[k];
  double * o = out + k * 4 * K;
  spherical_harmonics<L, true, double>(a.pair_dir[3 * p], a.pair_dir[3 * p + 1], a.pair_dir[3 * p + 2],
                                       [&](int lm, double y, double gx, double gy, double gz) {
                                         o[lm] = y;
                                         o[K + lm] = gx;
                                         o[2 * K + lm] = gy;
                                         o[3 * K + lm] = gz;
                                       });
}

template <int L>
void ps_bwd_f64(const PsArgs & ps, const double * C, const double * X, const double * inv_norm, const double * t,
                double * dC, cudaStream_t st) {
  const FeatureDims & fd = ps.fd;
  const int pnn = fd.P * fd.n * fd.n;
  // a row that only fits without the padding (what the forward needs) goes
  // unpadded
  const size_t need = sizeof(double) * (size_t(fd.Sn) * fd.K + fd.D);
  size_t smem = need + sizeof(double) * size_t(fd.L + 1) * (l_plane(pnn) - pnn);
  int plane = l_plane(pnn);
  if (smem > size_t(227) * 1024 - 1024) {
    smem = need;
    plane = pnn;
  }
  RGPU_CUDA(cudaFuncSetAttribute(ps_bwd_f64_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  ps_bwd_f64_kernel<L><<<unsigned(ps.n_centers), kBwdThreads, smem, st>>>(ps, plane, C, X, inv_norm, t, dC);
}

}  // namespace

#define RGPU_ADJ64_SWITCH(L_, CASE)                                                              \
  switch (L_) {                                                                                  \
    CASE(0) CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10)     \
    CASE(11) CASE(12)                                                                            \
    default:                                                                                     \
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_angular above 12 is not supported on the GPU"); \
  }

void launch_ps_bwd_fp64(const PsArgs & ps, const double * C, const double * X, const double * inv_norm,
                        const double * t, double * dC, cudaStream_t st) {
  if (ps.n_centers == 0) return;
#define RGPU_CASE(LL)                                \
  case LL:                                           \
    ps_bwd_f64<LL>(ps, C, X, inv_norm, t, dC, st); \
    break;
  RGPU_ADJ64_SWITCH(ps.fd.L, RGPU_CASE)
#undef RGPU_CASE
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

void launch_pair_adjoint_fp64(const ExpansionArgs & a, const double * dC, const int32_t * pair_center,
                              int64_t n_pairs, double * F, const int32_t * center_struct, double * stress,
                              cudaStream_t st) {
  if (a.n_centers == 0 || n_pairs == 0) return;
  sph_constants_tu();
  const unsigned grid = unsigned((n_pairs + kPairThreads - 1) / kPairThreads);
#define RGPU_CASE(LL)                                                                                             \
  case LL:                                                                                                        \
    pair_adjoint_f64_kernel<LL><<<grid, kPairThreads, 0, st>>>(a, pair_center, n_pairs, dC, F, center_struct, stress); \
    break;
  RGPU_ADJ64_SWITCH(a.fd.L, RGPU_CASE)
#undef RGPU_CASE
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

void launch_pair_harmonics_fp64(const ExpansionArgs & a, int64_t n, const int32_t * list, double * out,
                                cudaStream_t st) {
  if (n <= 0) return;
  sph_constants_tu();
  const unsigned grid = unsigned((n + kPairThreads - 1) / kPairThreads);
#define RGPU_CASE(LL)                                                          \
  case LL:                                                                     \
    pair_harmonics_kernel<LL><<<grid, kPairThreads, 0, st>>>(a, n, list, out); \
    break;
  RGPU_ADJ64_SWITCH(a.fd.L, RGPU_CASE)
#undef RGPU_CASE
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

}  // namespace rgpu
