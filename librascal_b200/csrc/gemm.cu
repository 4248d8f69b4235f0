// Dense contractions of the GAP model.
//
// Forward, per central species s:  k = X_s T_s^T,  e_i = sum_m alpha_m k^zeta,
// W = alpha zeta k^(zeta-1)   (models/sparse_kernels.hh:104-131,
// models/sparse_kernel_predict.hh:130-145, models/kernels.hh:48-61).
// Backward: dE/dX_s = W T_s (the "sparse_point_scaled" contraction of
// models/sparse_kernel_predict.hh:141-143, done for all centres at once).
//
// Two implementations:
//  * FP64 tensor-core tiles for the plain path (dgemm.cuh);
//  * TF32 tensor-core tiles (mma.sync m16n8k8) with FP32 accumulation for
//    the fast path, optionally as a 3-term split (hi*hi + hi*lo + lo*hi) that
//    carries ~21 mantissa bits. The forward epilogue fuses k^zeta, the
//    per-row energy partials and W, so k never touches HBM.
#include <cuda_runtime.h>

#include "common.cuh"
#include "dgemm.cuh"

namespace rgpu {
namespace {

__device__ __forceinline__ float pow_zeta_f(float v, int z) {
  float r = 1.f;
  for (int i = 0; i < z; ++i) r *= v;
  return r;
}

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

// ------------------------------------------------------ TF32 tensor-core GEMM
constexpr int kBM = 128, kBN = 128, kBKt = 32, kStages = 3, kLdS = kBKt + 4;
constexpr size_t kTf32Smem = size_t(kStages) * 2 * kBM * kLdS * sizeof(float);

__device__ __forceinline__ void cp_async16(void * smem, const void * gmem, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void mma_tf32(float * c, const uint32_t * a, const uint32_t * b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t tf32_bits(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

template <bool SPLIT>
__global__ void __launch_bounds__(256)
gemm_tf32_kernel(Tf32GemmArgs g) {
  extern __shared__ __align__(16) float sm[];
  float * As = sm;                                  // [stages][BM][LdS]
  float * Bs = sm + size_t(kStages) * kBM * kLdS;   // [stages][BN][LdS]
  __shared__ float row_e[kBM];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int wm = (wid >> 2) * 64, wn = (wid & 3) * 32;
  const int64_t n0 = int64_t(blockIdx.x) * kBN, m0 = int64_t(blockIdx.y) * kBM;
  if (g.epilogue == 1 && tid < kBM) row_e[tid] = 0.f;

  auto load_stage = [&](int stage, int64_t k0) {
    float * as = As + size_t(stage) * kBM * kLdS;
    float * bs = Bs + size_t(stage) * kBN * kLdS;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int idx = tid + q * 256;  // 1024 chunks of 16 B per operand
      int r = idx >> 3, cchunk = (idx & 7) * 4;
      int64_t ga = m0 + r;
      const float * src = g.A + (ga < g.M ? ga : 0) * g.lda + k0 + cchunk;
      cp_async16(as + r * kLdS + cchunk, src, ga < g.M ? 16 : 0);
      int64_t gb = n0 + r;
      const float * srcb = g.B + (gb < g.N ? gb : 0) * g.ldb + k0 + cchunk;
      cp_async16(bs + r * kLdS + cchunk, srcb, gb < g.N ? 16 : 0);
    }
  };

  float acc[4][4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[i][j][v] = 0.f;

  const int nk = int(g.K / kBKt);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nk) load_stage(s, int64_t(s) * kBKt);
    cp_commit();
  }
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<kStages - 2>();
    __syncthreads();
    {
      int nxt = kt + kStages - 1;
      if (nxt < nk) load_stage(nxt % kStages, int64_t(nxt) * kBKt);
      cp_commit();
    }
    const float * as = As + size_t(kt % kStages) * kBM * kLdS;
    const float * bs = Bs + size_t(kt % kStages) * kBN * kLdS;
#pragma unroll
    for (int kk = 0; kk < kBKt; kk += 8) {
      uint32_t ah[4][4], bh[4][2];
      uint32_t al[4][4], bl[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float * p = as + (wm + i * 16 + gid) * kLdS + kk + tig;
        float f[4] = {p[0], p[8 * kLdS], p[4], p[8 * kLdS + 4]};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          ah[i][v] = tf32_bits(f[v]);
          if (SPLIT) al[i][v] = tf32_bits(f[v] - __uint_as_float(ah[i][v]));
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float * p = bs + (wn + j * 8 + gid) * kLdS + kk + tig;
        float f[2] = {p[0], p[4]};
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          bh[j][v] = tf32_bits(f[v]);
          if (SPLIT) bl[j][v] = tf32_bits(f[v] - __uint_as_float(bh[j][v]));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (SPLIT) {
            mma_tf32(acc[i][j], al[i], bh[j]);
            mma_tf32(acc[i][j], ah[i], bl[j]);
          }
          mma_tf32(acc[i][j], ah[i], bh[j]);
        }
    }
  }
  cp_wait<0>();

  if (g.epilogue == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int64_t r = m0 + wm + i * 16 + gid + h * 8;
          int64_t c = n0 + wn + j * 8 + tig * 2;
          if (r < g.M && c < g.N) {
            float2 v = make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
            *reinterpret_cast<float2 *>(g.C + r * g.ldc + c) = v;
          }
        }
    return;
  }
  // GAP forward epilogue
  float re[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) re[i][0] = re[i][1] = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int64_t r = m0 + wm + i * 16 + gid + h * 8;
        int64_t c = n0 + wn + j * 8 + tig * 2;
        float w2[2];
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          float k = acc[i][j][2 * h + v];
          float al = (c + v < g.N) ? g.alpha[c + v] : 0.f;
          re[i][h] += al * pow_zeta_f(k, g.zeta);
          w2[v] = al * (float(g.zeta) * pow_zeta_f(k, g.zeta - 1));
        }
        if (r < g.M && c < g.ldc) *reinterpret_cast<float2 *>(g.C + r * g.ldc + c) = make_float2(w2[0], w2[1]);
      }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v = re[i][h];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      re[i][h] = v;
    }
  __syncthreads();
  if (tig == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) atomicAdd(&row_e[wm + i * 16 + gid + h * 8], re[i][h]);
  }
  __syncthreads();
  if (tid < kBM) {
    int64_t r = m0 + tid;
    if (r < g.M) g.e_part[int64_t(blockIdx.x) * g.M + r] = row_e[tid];
  }
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

bool g_tf32_split = true;

void gemm_tf32(const Tf32GemmArgs & g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0) return;
  if (g.K % kBKt != 0) throw Error(RGPU_ERR_INVALID_ARGUMENT, "TF32 GEMM: K must be a multiple of 32");
  dim3 grid(div_up(g.N, kBN), div_up(g.M, kBM));
  if (g_tf32_split) {
    RGPU_CUDA(cudaFuncSetAttribute(gemm_tf32_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(kTf32Smem)));
    gemm_tf32_kernel<true><<<grid, 256, kTf32Smem, st>>>(g);
  } else {
    RGPU_CUDA(cudaFuncSetAttribute(gemm_tf32_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(kTf32Smem)));
    gemm_tf32_kernel<false><<<grid, 256, kTf32Smem, st>>>(g);
  }
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
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
