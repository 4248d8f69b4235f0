// Adjoint force kernel of the fast path.
//
// Given dE/dc^i (from the power-spectrum backward), the force contribution of
// pair (i, j) is g_ij = sum_{n,lm} dE/dc^i_{type_j, n lm} * d c^i_{n lm}/d r_j,
// where d c^i / d r_j = (dRI f_c + RI df_c) Y r^ + RI f_c / r grad Y is
// recomputed here from the spline and the spherical-harmonics recurrence
// instead of being stored (the reference materialises it per pair,
// calculator_spherical_expansion.hh:2306-2366, and contracts it in
// models/sparse_kernel_predict.hh:147-172). The contraction is reordered as
//   g = r^ * sum_lm A_lm Y_lm + f_c / r * sum_lm B_lm grad Y_lm,
//   A_lm = sum_n E_{n lm} (dRI f_c + RI df_c)_{n l},  B_lm = sum_n E_{n lm} RI_{n l}.
// Forces follow the reference's accumulation (sparse_kernel_predict.hh:
// 257-263): F_j -= g_ij for every pair (folded onto the real atom) and
// F_i += g_ij unless j is a periodic image of i (the rule of
// calculator_spherical_expansion.hh:2354-2358).
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

#ifndef RGPU_ADJ_L0
#define RGPU_ADJ_L0 0
#define RGPU_ADJ_L1 12
#define RGPU_ADJ_DISPATCH
#endif

namespace rgpu {
namespace {

constexpr int kThreads = 128;
constexpr int kMaxN = 16;  // largest max_radial of the register-staged path
// Shared memory a block may take: four blocks of 128 threads stay resident.
constexpr size_t kBlockBytes = 72 * 1024;

// Floats between staged dE/dc rows: whole 16-byte units and one more, so that
// rows start in different banks.
__host__ __device__ constexpr int staged_row(int row_len) { return ((row_len + 3) & ~3) + 4; }

// One thread per pair (pairs of many centres share a warp, so no lane idles
// when centres have few neighbours); per l, the harmonics stream past the n
// radial values RI and p1 = dRI f_c + RI df_c in registers (NV >= n of them).
// The harmonics are polynomials q_lm(z) (x + iy)^m of the unit vector, whose z
// derivative is the next order's q, and whose plain gradient sum is projected
// onto the sphere once per pair at the end.
//
// Two reads would bound this kernel if each lane made its own, and a warp or
// block shares both:
//  - dE/dc of the centre, n (l+1)^2 values per pair, n contiguous ones per lm:
//    each waits on L1 or L2 with about 20 warps per SM to hide it. With STAGE
//    the rows of the block's centres (`rows` at a time) are copied to shared
//    memory first, every copy in flight at once. That pays while a block spans
//    few centres; the launch decides (10 000 clusters with 12 neighbours and
//    7.8 KB rows read theirs through L2, after a prefetch).
//  - the spline table: every pair lies in another interval, so 32 lanes read
//    32 lines per channel (30 wavefronts a load, half of the LSU's time). 8 or
//    4 lanes copy neighbouring channels of one pair's interval to shared
//    memory, asynchronously and one l ahead, and its own lane reads them there.
// What is left is issue: 1.6 instructions a cycle with 12 warps per SM.
// The loop over l is rolled: unrolled it outgrows the instruction cache (2.2 of
// 15 cycles per instruction wait for it). FULL (n = NV) keeps the bounds of
// the channel loops and the strides of 16-byte reads out of it.
// Each lane on its own and shared: 100 000 atoms with 46 neighbours at n = 12,
// l = 9, 4.2 and 1.9 ms; 10 000 clusters (n = 8, l = 6, 5 species) 1.04 and 0.64 ms; a box of
// 150 atoms with 34 neighbours (n = 8, l = 6) 26 and 13.6 us; 97 cells at
// n = 7, l = 5, 384 and 254 us.
//
// With `stress`, the pair's r_ji (x) g_ij (Voigt xx yy zz yz xz xy, the
// reference's sparse_kernel_predict.hh:355-366) is summed per structure as
// well. With `scale`, each structure's contributions are multiplied by
// scale[structure] (an upstream gradient; a pass of its own over dE/dc took
// 114 us for 16 000 atoms).
template <int L, int NV, bool FULL, bool STAGE>
__global__ void __launch_bounds__(kThreads, NV <= 8 ? 5 : 4)
pair_adjoint_kernel(ExpansionArgs a, const int32_t * __restrict__ pair_center, int64_t n_pairs,
                    const float * __restrict__ dC, double * __restrict__ F,
                    const int32_t * __restrict__ center_struct, double * __restrict__ stress,
                    const double * __restrict__ scale, int rows) {
  constexpr int L1 = L + 1, K = L1 * L1, SL = kMaxL + 2;
  extern __shared__ __align__(16) float sma[];
  const int W = a.fd.W, n = FULL ? NV : a.fd.n, Sn = a.fd.S * n;
  const int lane = threadIdx.x & 31;
  const int row_len = Sn * K, row_step = staged_row(row_len);
  constexpr int kRow = NV + 1;  // 16-byte units of a pair's spline row: odd, so that lanes meet different banks
  const float ih = float(a.sp.inv_h);
  const int warps = blockDim.x >> 5;
  float4 * tile = reinterpret_cast<float4 *>(sma) + (threadIdx.x >> 5) * 32 * kRow;
  float * staged = sma + 4 * warps * 32 * kRow;
  if (!FULL) {  // the channels past n stay zero
    for (int e = threadIdx.x; e < warps * 32 * kRow; e += blockDim.x)
      reinterpret_cast<float4 *>(sma)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
  }
  // the copies of this lane: channels c, c + kLanes, .. of every kLanes-th pair
  constexpr int kLanes = NV % 8 == 0 ? 8 : 4;
  const int mine = lane / kLanes, ch = lane % kLanes;
  const uint32_t tile_dst = static_cast<uint32_t>(__cvta_generic_to_shared(tile + mine * kRow + ch));
  const bool last_channel = NV - kLanes + ch < n;
  const uint32_t staged_dst = static_cast<uint32_t>(__cvta_generic_to_shared(staged));
  auto stage = [&](int32_t c_lo, int32_t c_hi) {
    for (int32_t c = c_lo; c < c_hi; ++c) {
      const float * src = dC + size_t(c) * row_len;
      const uint32_t dst = staged_dst + 4u * uint32_t((c - c_lo) * row_step);
      if (FULL || (row_len & 3) == 0) {
        for (int e = threadIdx.x; e < row_len / 4; e += blockDim.x)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + 4 * e) : "memory");
      } else {
        for (int e = threadIdx.x; e < row_len; e += blockDim.x)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * e), "l"(src + e) : "memory");
      }
    }
  };
  // the list's own total bounds the loop (below n_pairs when the list was
  // built to a capacity)
  {
    const int64_t listed = a.pair_off[a.n_centers];
    if (listed < n_pairs) n_pairs = listed;
  }
  // the loop bound is uniform over the block: its warps stage rows together
  // and their lanes shuffle below
  for (int64_t base = int64_t(blockIdx.x) * blockDim.x; base < n_pairs; base += int64_t(gridDim.x) * blockDim.x) {
    const int64_t p = base + threadIdx.x;
    const int32_t ci = p < n_pairs ? pair_center[p] : -1;
    int32_t c_first = 0, c_last = 0;  // the block's centres
    if (STAGE) {
      c_first = pair_center[base];
      c_last = pair_center[min(base + int64_t(blockDim.x), n_pairs) - 1];
      __syncthreads();  // the rows staged before are read no more
      stage(c_first, min(c_last + 1, c_first + rows));
    } else {
      // the lanes of one centre bring its dE/dc row (Sn K floats, read
      // below one lm at a time) towards L2 together, before the spline and
      // Y_lm work, so that the reads below wait on L2 rather than DRAM
      const unsigned same = __match_any_sync(0xffffffffu, ci);
      if (ci >= 0) {
        const int rank = __popc(same & lanemask_lt()), run = __popc(same);
        const char * line = reinterpret_cast<const char *>(dC + size_t(ci) * row_len);
        const int lines = (row_len * 4 + 127) >> 7;
        for (int k = rank; k < lines; k += run)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(line + (size_t(k) << 7)));
      }
    }
    // the self pair carries no force of its own (the other pairs' F_i terms
    // do); it and the lanes past the list go along with nothing to add
    const bool own = ci >= 0 && p != a.pair_off[ci];
    float g0 = 0.f, g1 = 0.f, g2 = 0.f, x = 0.f, y = 0.f, z = 1.f, rf = 1.f, fc = 0.f, dfc = 0.f;
    int32_t j = -1, self_atom = -1;
    int col = 0;  // the neighbour's species in a dE/dc row
    float aa = 1.f, bb = 0.f;
    int interval = 0;
    if (own) {
      self_atom = a.center_atom[ci];
      const double r = a.pair_dist[p];
      j = a.pair_j[p];
      col = a.species_lut[a.types[j]] * n;
      double fcd, dfcd;
      cutoff_fc_dfc(a, r, fcd, dfcd);
      fc = float(fcd);
      dfc = float(dfcd);
      const SplinePos q = spline_pos(a.sp, r);
      aa = float(q.a);
      bb = float(q.b);
      interval = q.k;
      x = float(a.pair_dir[3 * p]);
      y = float(a.pair_dir[3 * p + 1]);
      z = float(a.pair_dir[3 * p + 2]);
      rf = float(r);
    }
    const float ca = aa * aa - 1.f, cb = bb * bb - 1.f;
    const float ea = 3.f * aa * aa - 1.f, eb = 3.f * bb * bb - 1.f;
    // interval k of the spline: (y_k, y2h_k, y_k+1, y2h_k+1) per channel
    uint32_t from[kLanes];
#pragma unroll
    for (int k = 0; k < kLanes; ++k)
      from[k] = uint32_t(__shfl_sync(0xffffffffu, interval, 32 / kLanes * k + mine)) * uint32_t(W) + uint32_t(ch);
    auto fetch = [&](int l) {
      const float4 * q4 = a.sp.q4f + l * n;
#pragma unroll
      for (int k = 0; k < kLanes; ++k)
#pragma unroll
        for (int c = 0; c < NV; c += kLanes)
          if (c + kLanes < NV || last_channel)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                             tile_dst + 16 * (32 / kLanes * k * kRow + c)),
                         "l"(q4 + from[k] + c)
                         : "memory");
    };
    for (int32_t c_lo = c_first; c_lo <= c_last; c_lo += STAGE ? rows : 1) {
      const int32_t c_hi = STAGE ? min(c_last + 1, c_lo + rows) : 1;
      const bool here = own && (!STAGE || (ci >= c_lo && ci < c_hi));
      const bool any = __any_sync(0xffffffffu, here);
      if (STAGE && c_lo != c_first) {
        __syncthreads();
        stage(c_lo, c_hi);
      }
      if (any) fetch(0);
      if (STAGE) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
      }
      if (!any) continue;
      const float * E = STAGE ? staged : dC;  // any row will do for the lanes without a pair here
      if (here) E += (STAGE ? (ci - c_lo) * size_t(row_step) : ci * size_t(row_len)) + col;
      float re[L1], im[L1];  // (x + iy)^m
      re[0] = 1.f;
      im[0] = 0.f;
#pragma unroll
      for (int m = 1; m <= L; ++m) {
        re[m] = re[m - 1] * x - im[m - 1] * y;
        im[m] = re[m - 1] * y + im[m - 1] * x;
      }
      float q1[L1], q0[L1 + 1];  // q of l - 1 and l
#pragma unroll
      for (int m = 0; m <= L; ++m) q0[m] = q1[m] = 0.f;
      q0[L1] = 0.f;
      float sY = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
      float cmm = 0.398942280401432677939946059934381868f;  // sqrt(1/(2 pi))
#pragma unroll 1
      for (int l = 0; l <= L; ++l) {
        // q_lm: the recursion in l (math/spherical_harmonics.cc:54-91), q_mm
        if (l > 0) cmm *= SphC<float>::c2(l);
#pragma unroll
        for (int m = 0; m <= L; ++m) {
          if (m > l) break;
          float v;
          if (m == l)
            v = cmm;
          else if (m == l - 1)
            v = SphC<float>::c1(l) * z * q0[m];
          else
            v = (z * q0[m] + SphC<float>::b(l * SL + m) * q1[m]) * SphC<float>::a(l * SL + m);
          q1[m] = q0[m];
          q0[m] = v;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();  // the warp's spline values of this l have landed
        float rl[NV], pl[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          const float4 t = tile[lane * kRow + k];
          const float ri = aa * (t.x + ca * t.y) + bb * (t.z + cb * t.w);
          const float dri = (t.z - t.x - ea * t.y + eb * t.w) * ih;
          rl[k] = ri;
          pl[k] = dri * fc + ri * dfc;
        }
        __syncwarp();  // and are read: the next l's may follow
        if (l < L) fetch(l + 1);
        auto dots = [&](int lm, float & A, float & B) {
          A = 0.f;
          B = 0.f;
          if (FULL) {
            const float4 * E4 = reinterpret_cast<const float4 *>(E + lm * Sn);
#pragma unroll
            for (int k = 0; k < NV / 4; ++k) {
              const float4 e = STAGE ? E4[k] : __ldg(E4 + k);
              A = fmaf(e.w, pl[4 * k + 3], fmaf(e.z, pl[4 * k + 2], fmaf(e.y, pl[4 * k + 1], fmaf(e.x, pl[4 * k], A))));
              B = fmaf(e.w, rl[4 * k + 3], fmaf(e.z, rl[4 * k + 2], fmaf(e.y, rl[4 * k + 1], fmaf(e.x, rl[4 * k], B))));
            }
          } else {
#pragma unroll
            for (int k = 0; k < NV; ++k)
              if (k < NV - 3 || k < n) {  // NV is n rounded up to a multiple of 4
                const float e = STAGE ? E[lm * Sn + k] : __ldg(E + lm * Sn + k);
                A = fmaf(e, pl[k], A);
                B = fmaf(e, rl[k], B);
              }
          }
        };
        const int o = l * l + l;
#pragma unroll
        for (int m = 0; m <= L; ++m) {
          if (m > l) break;
          // dq_lm/dz = -sqrt((l - m)(l + m + 1)) q_l,m+1
          const float dq = m < l ? -SphC<float>::plm(l * SL + m) * q0[m + 1] : 0.f;
          float A, B;
          dots(o + m, A, B);
          if (m == 0) {
            constexpr float kInvSqrt2 = 0.707106781186547524400844362104849039f;
            sY = fmaf(A, q0[0] * kInvSqrt2, sY);
            sz = fmaf(B, dq * kInvSqrt2, sz);
          } else {
            float A2, B2;
            dots(o - m, A2, B2);
            const float tq = q0[m] * float(m), c = tq * re[m - 1], d = tq * im[m - 1];
            sY = fmaf(q0[m], fmaf(A, re[m], A2 * im[m]), sY);
            sx += fmaf(B, c, B2 * d);
            sy += fmaf(B2, c, -B * d);
            sz = fmaf(dq, fmaf(B, re[m], B2 * im[m]), sz);
          }
        }
      }
      if (here) {
        // the tangential part of the gradient sum
        const float along = x * sx + y * sy + z * sz, fr = fc / rf;
        const float up = scale ? float(scale[center_struct[ci]]) : 1.f;
        g0 = up * (x * sY + fr * (sx - x * along));
        g1 = up * (y * sY + fr * (sy - y * along));
        g2 = up * (z * sY + fr * (sz - z * along));
        atomicAdd(&F[3 * size_t(j) + 0], -double(g0));
        atomicAdd(&F[3 * size_t(j) + 1], -double(g1));
        atomicAdd(&F[3 * size_t(j) + 2], -double(g2));
      }
    }
    // F_i += g unless j is a periodic image of i: the centre's pairs are
    // consecutive lanes, so a segmented warp scan leaves each run's sum in
    // its last lane and one atomic per run and component remains.
    const bool other = j >= 0 && j != self_atom;
    float h0 = other ? g0 : 0.f, h1 = other ? g1 : 0.f, h2 = other ? g2 : 0.f;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float u0 = __shfl_up_sync(0xffffffffu, h0, off);
      const float u1 = __shfl_up_sync(0xffffffffu, h1, off);
      const float u2 = __shfl_up_sync(0xffffffffu, h2, off);
      const int32_t cu = __shfl_up_sync(0xffffffffu, ci, off);
      if (lane >= off && cu == ci) {
        h0 += u0;
        h1 += u1;
        h2 += u2;
      }
    }
    const int32_t cn = __shfl_down_sync(0xffffffffu, ci, 1);
    if (ci >= 0 && (lane == 31 || cn != ci)) {
      const int32_t ia = a.center_atom[ci];
      atomicAdd(&F[3 * size_t(ia) + 0], double(h0));
      atomicAdd(&F[3 * size_t(ia) + 1], double(h1));
      atomicAdd(&F[3 * size_t(ia) + 2], double(h2));
    }
    if (stress) {
      const float rx = -rf * x, ry = -rf * y, rz = -rf * z;  // g is zero without a pair of its own
      float t6[6] = {rx * g0, ry * g1, rz * g2, ry * g2, rz * g0, rx * g1};
      // structures are consecutive runs of centres, hence of lanes
      const int32_t sid = ci >= 0 ? center_struct[ci] : -1;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int32_t su = __shfl_up_sync(0xffffffffu, sid, off);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          const float u = __shfl_up_sync(0xffffffffu, t6[k], off);
          if (lane >= off && su == sid) t6[k] += u;
        }
      }
      const int32_t sn = __shfl_down_sync(0xffffffffu, sid, 1);
      if (sid >= 0 && (lane == 31 || sn != sid))
#pragma unroll
        for (int k = 0; k < 6; ++k) atomicAdd(&stress[6 * size_t(sid) + k], double(t6[k]));
    }
  }
}

// One instantiation per (L, NV): compiled in the translation unit that owns
// L (the library builds this file once per range of L, in parallel, since
// each instantiation unrolls the spherical-harmonics recurrence).
template <int L, int NV>
void adjoint_launch_nv(const ExpansionArgs & a, const int32_t * pair_center, int64_t n_pairs, const float * dC,
                       double * forces, cudaStream_t st, const int32_t * center_struct, double * stress,
                       const double * scale, int grid, int threads) {
  // rows of the centres a block of pairs spans on average, and two more; a
  // block that spans others takes them in turn
  const size_t row = sizeof(float) * staged_row(a.fd.Sn * a.fd.K);
  const int64_t per_centre = std::max<int64_t>(1, a.n_pairs / a.n_centers);
  const int rows = int(threads / per_centre) + 2;
  const size_t own = 16 * size_t(threads) * (NV + 1);
  const bool stage = own + rows * row <= kBlockBytes;
  const bool full = a.fd.n == NV;
  const auto kernel = full ? (stage ? pair_adjoint_kernel<L, NV, true, true> : pair_adjoint_kernel<L, NV, true, false>)
                           : (stage ? pair_adjoint_kernel<L, NV, false, true> : pair_adjoint_kernel<L, NV, false, false>);
  RGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBlockBytes)));
  kernel<<<grid, threads, stage ? own + rows * row : own, st>>>(a, pair_center, n_pairs, dC, forces, center_struct,
                                                              stress, scale, rows);
}

template <int L>
void adjoint_launch(const ExpansionArgs & a, const int32_t * pair_center, int64_t n_pairs, const float * dC,
                    double * forces, cudaStream_t st, const int32_t * center_struct, double * stress,
                    const double * scale, int grid, int threads) {
  sph_constants_tu();  // this translation unit's copy of the constants
  if (a.fd.n <= 4)
    adjoint_launch_nv<L, 4>(a, pair_center, n_pairs, dC, forces, st, center_struct, stress, scale, grid, threads);
  else if (a.fd.n <= 8)
    adjoint_launch_nv<L, 8>(a, pair_center, n_pairs, dC, forces, st, center_struct, stress, scale, grid, threads);
  else if (a.fd.n <= 12)
    adjoint_launch_nv<L, 12>(a, pair_center, n_pairs, dC, forces, st, center_struct, stress, scale, grid, threads);
  else
    adjoint_launch_nv<L, 16>(a, pair_center, n_pairs, dC, forces, st, center_struct, stress, scale, grid, threads);
}

}  // namespace

// Launch of the adjoint kernels of one L. Each translation unit
// instantiates it for its own range of L (explicit instantiation below); the
// dispatch refers to the others through extern declarations.
template <int L>
void adjoint_launch_l(const ExpansionArgs & a, const int32_t * pc, int64_t np, const float * dC, double * F,
                      cudaStream_t st, const int32_t * cs, double * S, const double * scale, int grid, int threads) {
  adjoint_launch<L>(a, pc, np, dC, F, st, cs, S, scale, grid, threads);
}

#define RGPU_ADJ_SIG(LL)                                                                                  \
  void adjoint_launch_l<LL>(const ExpansionArgs &, const int32_t *, int64_t, const float *, double *,     \
                            cudaStream_t, const int32_t *, double *, const double *, int, int)
#define RGPU_ADJ_INST(LL)                                             \
  template RGPU_ADJ_SIG(LL);
#define RGPU_ADJ_EXTERN(LL)                                           \
  extern template RGPU_ADJ_SIG(LL);
#if RGPU_ADJ_L0 <= 0 && 0 <= RGPU_ADJ_L1
RGPU_ADJ_INST(0)
#else
RGPU_ADJ_EXTERN(0)
#endif
#if RGPU_ADJ_L0 <= 1 && 1 <= RGPU_ADJ_L1
RGPU_ADJ_INST(1)
#else
RGPU_ADJ_EXTERN(1)
#endif
#if RGPU_ADJ_L0 <= 2 && 2 <= RGPU_ADJ_L1
RGPU_ADJ_INST(2)
#else
RGPU_ADJ_EXTERN(2)
#endif
#if RGPU_ADJ_L0 <= 3 && 3 <= RGPU_ADJ_L1
RGPU_ADJ_INST(3)
#else
RGPU_ADJ_EXTERN(3)
#endif
#if RGPU_ADJ_L0 <= 4 && 4 <= RGPU_ADJ_L1
RGPU_ADJ_INST(4)
#else
RGPU_ADJ_EXTERN(4)
#endif
#if RGPU_ADJ_L0 <= 5 && 5 <= RGPU_ADJ_L1
RGPU_ADJ_INST(5)
#else
RGPU_ADJ_EXTERN(5)
#endif
#if RGPU_ADJ_L0 <= 6 && 6 <= RGPU_ADJ_L1
RGPU_ADJ_INST(6)
#else
RGPU_ADJ_EXTERN(6)
#endif
#if RGPU_ADJ_L0 <= 7 && 7 <= RGPU_ADJ_L1
RGPU_ADJ_INST(7)
#else
RGPU_ADJ_EXTERN(7)
#endif
#if RGPU_ADJ_L0 <= 8 && 8 <= RGPU_ADJ_L1
RGPU_ADJ_INST(8)
#else
RGPU_ADJ_EXTERN(8)
#endif
#if RGPU_ADJ_L0 <= 9 && 9 <= RGPU_ADJ_L1
RGPU_ADJ_INST(9)
#else
RGPU_ADJ_EXTERN(9)
#endif
#if RGPU_ADJ_L0 <= 10 && 10 <= RGPU_ADJ_L1
RGPU_ADJ_INST(10)
#else
RGPU_ADJ_EXTERN(10)
#endif
#if RGPU_ADJ_L0 <= 11 && 11 <= RGPU_ADJ_L1
RGPU_ADJ_INST(11)
#else
RGPU_ADJ_EXTERN(11)
#endif
#if RGPU_ADJ_L0 <= 12 && 12 <= RGPU_ADJ_L1
RGPU_ADJ_INST(12)
#else
RGPU_ADJ_EXTERN(12)
#endif
#undef RGPU_ADJ_EXTERN
#undef RGPU_ADJ_INST
#undef RGPU_ADJ_SIG

#ifdef RGPU_ADJ_DISPATCH
void launch_pair_adjoint_fp32(const ExpansionArgs & a, const int32_t * pair_center, int64_t n_pairs,
                              const float * dC, double * forces, cudaStream_t st,
                              const int32_t * center_struct, double * stress, const double * scale) {
  if (a.n_centers == 0 || n_pairs == 0) return;
  if (a.fd.n > kMaxN) throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_radial above 16 is not supported on the fast path");
  const TileConfig cfg = tile_config(a.fd.S, a.fd.n, a.fd.L);
  const int threads = std::min(cfg.adj_threads, kThreads);
  int dev = 0, sms = 148;
  RGPU_CUDA(cudaGetDevice(&dev));
  RGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid =
      int(std::min<int64_t>((n_pairs + threads - 1) / threads, int64_t(sms) * cfg.adj_blocks_per_sm));
#define RGPU_ADJ_CASE(LL)                                                                        \
  case LL:                                                                                       \
    adjoint_launch_l<LL>(a, pair_center, n_pairs, dC, forces, st, center_struct, stress, scale, grid, threads); \
    break;
  switch (a.fd.L) {
    RGPU_ADJ_CASE(0)
    RGPU_ADJ_CASE(1)
    RGPU_ADJ_CASE(2)
    RGPU_ADJ_CASE(3)
    RGPU_ADJ_CASE(4)
    RGPU_ADJ_CASE(5)
    RGPU_ADJ_CASE(6)
    RGPU_ADJ_CASE(7)
    RGPU_ADJ_CASE(8)
    RGPU_ADJ_CASE(9)
    RGPU_ADJ_CASE(10)
    RGPU_ADJ_CASE(11)
    RGPU_ADJ_CASE(12)
    default:
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_angular above 12 is not supported on the GPU");
  }
#undef RGPU_ADJ_CASE
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}
#endif

}  // namespace rgpu
