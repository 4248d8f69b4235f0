// FP64 tile GEMM on the tensor cores (mma.sync m16n8k8 f64): C[r][c] =
// sum_k A[r][k] B(k, c), the result handed to an epilogue functor (what a row
// needs is looked up once per row). B is either N x K row-major (B_NT,
// C = A B^T) or K x N row-major. Several problems (one per species) run in
// one launch, and K can be cut into splits whose partial sums go to separate
// planes that the caller's next kernel adds.
//
// What bounds it: the FP64 tensor pipe (37.0 TFLOP/s measured with register
// operands, peaks.cu; FMA chains reach 34.2), which only a full grid reaches.
// The tile is 64 x 64 rather than 128 x 128 because a warp's 32 x 32 part of it
// reads 64 doubles per 1024 FMAs, which shared memory delivers in time, and
// because the GAP contractions are ragged: per species a few hundred to a few
// thousand rows by 50..2000 sparse points. 128 x 128 tiles of one species at a
// time left 6 to 84 blocks on 148 SMs. Splits of K fill the chip where even
// 64 x 64 tiles of every species do not.
//
// 128 threads, 2 x 2 warps of 32 x 32; slices of 16 k in a three-deep
// cp.async ring. The shared row strides (20 doubles for k-major tiles, 68
// for the K x N tile, both 4 modulo 16) put the 16 operands of a half-warp
// load in 16 different 8-byte banks.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace rgpu {

constexpr int kDgBM = 64, kDgBN = 64, kDgBK = 16, kDgStages = 3, kDgThreads = 128;
constexpr int kDgLdK = kDgBK + 4, kDgLdN = kDgBN + 4;  // shared row strides, in doubles
constexpr int kDgStageA = kDgBM * kDgLdK;
constexpr int kDgStageB = kDgBN * kDgLdK;  // covers the 16 x 68 tile too
constexpr size_t kDgSmem = sizeof(double) * kDgStages * (kDgStageA + kDgStageB);
constexpr int kDgMaxProblems = kMaxSpecies;
static_assert(kDgBK * kDgLdN <= kDgStageB, "the K x N tile fits the stage");

// C[split][r][c]; planes are `plane` values apart.
struct DgStoreC {
  double * C;
  int64_t ldc, plane;
  __device__ __forceinline__ double * row(int64_t r) const { return C + r * ldc; }
  __device__ __forceinline__ void put(double * o, int c, double v, int split) const { o[split * plane + c] = v; }
};

template <class Epi>
struct DgProblem {
  int64_t M;
  int N, K;
  const double * A;
  int64_t lda;
  const double * B;
  int64_t ldb;
  Epi epi;
};
template <class Epi>
struct DgGroup {
  int n, splits;
  int64_t tile_end[kDgMaxProblems];  // running tile counts
  DgProblem<Epi> p[kDgMaxProblems];
};

__device__ __forceinline__ void dg_cp(double * smem, const double * gmem, int bytes, int full) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  // bytes < full: the rest is filled with zeros
  if (full == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dmma(double * c, const double * a, const double * b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// VEC: doubles per copy, 2 when every row of both operands starts on a
// 16-byte boundary, else 1.
template <bool B_NT, int VEC, class Epi>
__global__ void __launch_bounds__(kDgThreads)
dgemm_kernel(const __grid_constant__ DgGroup<Epi> g) {
  extern __shared__ __align__(16) double dsm[];
  constexpr int kFull = 8 * VEC;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int split = int(blockIdx.x % unsigned(g.splits));
  const int64_t tile = blockIdx.x / unsigned(g.splits);
  int pi = 0;
  while (tile >= g.tile_end[pi]) ++pi;
  const DgProblem<Epi> & p = g.p[pi];
  const int64_t local = tile - (pi ? g.tile_end[pi - 1] : 0);
  // column tiles vary fastest: the blocks that share an A row tile run
  // together, so A comes from DRAM once and the others read it from L2
  const int tiles_n = (p.N + kDgBN - 1) / kDgBN;
  const int64_t r0 = local / tiles_n * kDgBM;
  const int c0 = int(local % tiles_n) * kDgBN;
  const int slices = (p.K + kDgBK - 1) / kDgBK, per = (slices + g.splits - 1) / g.splits;
  const int k_lo = min(split * per, slices) * kDgBK, k_hi = min(min((split + 1) * per, slices) * kDgBK, p.K);

  // copies: `kRow` threads side by side on a row of 16 k, rows kRows apart
  constexpr int kRow = kDgBK / VEC, kRows = kDgThreads / kRow, kCopies = kDgBM / kRows;
  const int lr = t / kRow, lk = (t % kRow) * VEC;
  int64_t a_off[kCopies], b_off[kCopies];
#pragma unroll
  for (int q = 0; q < kCopies; ++q) {
    const int64_t r = r0 + lr + q * kRows;
    a_off[q] = r < p.M ? r * p.lda : int64_t(-1);
    const int c = c0 + lr + q * kRows;
    b_off[q] = c < p.N ? int64_t(c) * p.ldb : int64_t(-1);
  }
  // the K x N tile: kCol threads side by side on a row of 64 columns
  constexpr int kCol = kDgBN / VEC, kColRows = kDgThreads / kCol, kColCopies = kDgBK / kColRows;
  const int nk = t / kCol, nc = (t % kCol) * VEC;

  auto load = [&](int stage, int k0) {
    double * as = dsm + stage * (kDgStageA + kDgStageB);
    double * bs = as + kDgStageA;
    const int kb = max(0, min(kFull, 8 * (k_hi - (k0 + lk))));
#pragma unroll
    for (int q = 0; q < kCopies; ++q) {
      const int n = a_off[q] >= 0 ? kb : 0;
      dg_cp(as + (lr + q * kRows) * kDgLdK + lk, n ? p.A + a_off[q] + k0 + lk : p.A, n, kFull);
    }
    if (B_NT) {
#pragma unroll
      for (int q = 0; q < kCopies; ++q) {
        const int n = b_off[q] >= 0 ? kb : 0;
        dg_cp(bs + (lr + q * kRows) * kDgLdK + lk, n ? p.B + b_off[q] + k0 + lk : p.B, n, kFull);
      }
    } else {
      const int cb = max(0, min(kFull, 8 * (p.N - (c0 + nc))));
#pragma unroll
      for (int q = 0; q < kColCopies; ++q) {
        const int k = k0 + nk + q * kColRows;
        const int n = k < k_hi ? cb : 0;
        dg_cp(bs + (nk + q * kColRows) * kDgLdN + nc, n ? p.B + int64_t(k) * p.ldb + c0 + nc : p.B, n, kFull);
      }
    }
  };

  double acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[i][j][v] = 0.;
  const int wm = (wid >> 1) * 32, wn = (wid & 1) * 32;
  const int iters = k_hi > k_lo ? (k_hi - k_lo + kDgBK - 1) / kDgBK : 0;
#pragma unroll
  for (int s = 0; s < kDgStages - 1; ++s) {
    if (s < iters) load(s, k_lo + s * kDgBK);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int stage = 0;
  for (int it = 0; it < iters; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kDgStages - 2) : "memory");
    __syncthreads();  // slice `it` has landed for every thread; the slice before it is read no more
    {
      const int nxt = it + kDgStages - 1;
      if (nxt < iters) load(nxt % kDgStages, k_lo + nxt * kDgBK);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const double * as = dsm + stage * (kDgStageA + kDgStageB);
    const double * bs = as + kDgStageA;
    stage = stage + 1 == kDgStages ? 0 : stage + 1;
#pragma unroll
    for (int kk = 0; kk < kDgBK; kk += 8) {
      double a[2][4], b[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double * q = as + (wm + 16 * i + gid) * kDgLdK + kk + tig;
        a[i][0] = q[0];
        a[i][1] = q[8 * kDgLdK];
        a[i][2] = q[4];
        a[i][3] = q[8 * kDgLdK + 4];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (B_NT) {
          const double * q = bs + (wn + 8 * j + gid) * kDgLdK + kk + tig;
          b[j][0] = q[0];
          b[j][1] = q[4];
        } else {
          const double * q = bs + (kk + tig) * kDgLdN + wn + 8 * j + gid;
          b[j][0] = q[0];
          b[j][1] = q[4 * kDgLdN];
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[i], b[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t r = r0 + wm + 16 * i + gid + 8 * h;
      if (r >= p.M) continue;
      const auto row = p.epi.row(r);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int c = c0 + wn + 8 * j + 2 * tig + v;
          if (c < p.N) p.epi.put(row, c, acc[i][j][2 * h + v], split);
        }
    }
}

// Splits of K that bring `tiles` tiles to about three blocks per SM (what
// the ring's shared memory lets be resident), each at least 4 slices deep.
inline int dgemm_splits(int64_t tiles, int K) {
  if (tiles <= 0) return 1;
  const int64_t want = std::max<int64_t>(1, 3 * 148 / tiles);
  return int(std::min<int64_t>({want, std::max(1, K / (4 * kDgBK)), 32}));
}
inline int64_t dgemm_tiles(int64_t M, int N) {
  return ((M + kDgBM - 1) / kDgBM) * int64_t((N + kDgBN - 1) / kDgBN);
}

// Launches the group (p[0..n) filled); `aligned` says that every row of A
// and B starts on a 16-byte boundary.
template <bool B_NT, class Epi>
void launch_dgemm(DgGroup<Epi> & g, bool aligned, cudaStream_t st) {
  int64_t tiles = 0;
  for (int i = 0; i < g.n; ++i) {
    tiles += dgemm_tiles(g.p[i].M, g.p[i].N);
    g.tile_end[i] = tiles;
  }
  if (tiles == 0) return;
  if (tiles * g.splits > 0x7fffffff) throw Error(RGPU_ERR_CAPACITY, "FP64 GEMM: too many rows for one launch");
  auto kernel = aligned ? dgemm_kernel<B_NT, 2, Epi> : dgemm_kernel<B_NT, 1, Epi>;
  RGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kDgSmem)));
  kernel<<<unsigned(tiles * g.splits), kDgThreads, kDgSmem, st>>>(g);
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

inline bool dgemm_aligned(const void * p, int64_t ld) {
  return (ld & 1) == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

}  // namespace rgpu
