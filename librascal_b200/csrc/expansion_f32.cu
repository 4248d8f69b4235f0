// FP32 spherical expansion (the FP64 one, in the reference's accumulation
// order, is expansion.cu): C[i][S n][row_stride(L)], each l-block padded to
// four floats, and the mask of the species among the centre's neighbours.
//
// Three kernels, by neighbours per centre and by the number of centres (see
// launch_expansion_fp32 and the constants below). With many neighbours: one
// warp per centre, pairs by species (pairs_f32.cuh). The coefficients of
// one species stay in registers, lanes over lm and n per lane, while its pairs
// pass: per pair and 32 lm one value of Y and n/4 broadcast loads of f_c RI
// feed n products. They are written once per species. Kept in global memory
// between chunks of 8 or 16 pairs they are 12.7 KB read and written per chunk
// at S = 2, n = 12, l = 9, some 15 GB for 100 000 atoms.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "pairs_f32.cuh"

namespace rgpu {
namespace {

constexpr int kMaxWarps = 8;
// Pairs per centre (self pairs included) from which the species-sorted kernel
// takes over. It wins once the coefficients would pass through global memory
// several times: 46 neighbours, S = 2, n = 12, l = 9 in chunks of 8: 3.95 ->
// 2.94 ms per 100 000 centres; 53 neighbours, S = 4, n = 7, l = 5: 0.42 ->
// 0.34 ms per 28 500. At 14 neighbours of 5 species (one chunk of 16) it took
// 1.11 ms against 0.84 per 161 000 centres (its sums are written species by
// species), and at 34 neighbours of 2 species 37 us against 33 per 2 000.
constexpr int64_t kFewPairs = 40;
// With one species the chunked kernel rewrites that species' sums alone, and
// the registers pay only where a lane has between 17 and 63 of them: few sums
// are cheap to rewrite, and from 64 on one block is resident per SM. Registers
// and chunks, ms, 20 000 centres with 65 neighbours: n = 8, l = 6 (16 sums)
// 0.35 and 0.31; n = 9, l = 8 (36) 0.74 and 0.71; n = 12, l = 9 (48) 0.88 and
// 1.00; n = 14, l = 10 (64) 1.96 and 1.50; n = 16, l = 12 (96) 2.62 and 2.05.
// With two species the two are within 5 % at both ends.
constexpr int kSumsLow = 16, kSumsHigh = 64;
// Centres per SM up to which a centre gets a block rather than a warp (warp
// and block, us): 1 000 centres of a box 30 and 22, 1 600 of 100 clusters 26
// and 22, 1 728 of a box at n = 12, l = 9 76 and 61; 2 000 of a box 33.5 and
// 33.6, 3 200 of 200 clusters 30 and 38.
constexpr int64_t kFewCentres = 12;

template <int L, int NV>
struct ExpSmem {
  using P = PairShape<L>;
  static constexpr int KP = P::K | 1;  // row stride of Y
  static constexpr int RI = P::L1 * NV;
  // floats per warp: the window's spline weights (4), x, y, z, k, species; Y
  // rows; radial rows
  static constexpr int kFloats = 9 * kWindow + (P::CH * KP + 3) / 4 * 4 + P::CH * RI;
  // Resident blocks of 256 threads the registers are cut for: three while
  // the accumulators are few (L = 6, n = 8: 16), two up to 48, else one.
  static constexpr int kBlocks = P::G * NV <= 32 ? 3 : (P::G * NV <= 48 ? 2 : 1);
};

template <int L, int NV>
__global__ void __launch_bounds__(kMaxWarps * 32, ExpSmem<L, NV>::kBlocks)
expansion_f32_kernel(ExpansionArgs a, float * __restrict__ C, uint32_t * __restrict__ present) {
  using P = PairShape<L>;
  using SM = ExpSmem<L, NV>;
  constexpr int K = P::K, L1 = P::L1, CH = P::CH, G = P::G, NL = P::NL, RS = row_stride(L), PAD = RS - K;
  extern __shared__ __align__(16) float smf[];
  __shared__ HarmonicConstants<L> hc;
  __shared__ int16_t dst_s[L1 * 16];  // channel (l, n) of the table -> place in a radial row
  __shared__ int16_t padc_s[PAD];     // columns of a padded row that belong to no (l, m)
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int W = a.fd.W, S = a.fd.S, n = a.fd.n;
  float4 * wt = reinterpret_cast<float4 *>(smf + wid * SM::kFloats);  // [kWindow]
  float * geo = reinterpret_cast<float *>(wt + kWindow);              // x, y, z [3][kWindow]
  int * gk = reinterpret_cast<int *>(geo + 3 * kWindow);              // spline interval
  int * gs = gk + kWindow;                                            // neighbour species
  float * Y = reinterpret_cast<float *>(gs + kWindow);
  float * R = Y + (CH * SM::KP + 3) / 4 * 4;
  hc.fill();
  for (int c = threadIdx.x; c < W; c += blockDim.x) dst_s[c] = int16_t(c / n * NV + c % n);
  for (int e = threadIdx.x; e < PAD; e += blockDim.x) {
    int left = e, l = 0;
    while (l <= L && left >= pad4(2 * l + 1) - (2 * l + 1)) {
      left -= pad4(2 * l + 1) - (2 * l + 1);
      ++l;
    }
    padc_s[e] = int16_t(l <= L ? offp_rt(l) + 2 * l + 1 + left : offp(L1) + left);
  }
  for (int e = lane; e < CH * SM::RI; e += 32) R[e] = 0.f;  // channels n .. NV-1 stay zero
  __syncthreads();
  int lg[G], col[G];  // this lane's l and padded column per group
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int lm = min(lane + 32 * g, K - 1);
    int l = 0;
#pragma unroll
    for (int q = 1; q <= L; ++q) l += lm >= q * q;
    lg[g] = l * NV;
    col[g] = offp_rt(l) + lm - l * l;
  }
  const int hq = lane / NL, hj = lane - hq * NL;  // this lane's pair and order in the harmonics
  for (int64_t ci = int64_t(blockIdx.x) * nw + wid; ci < a.n_centers; ci += int64_t(gridDim.x) * nw) {
    float * Ci = C + size_t(ci) * S * n * RS;
    const int64_t p_lo = a.pair_off[ci] + 1, p_hi = a.pair_off[ci + 1];
    const int ti = a.species_lut[a.types[a.center_atom[ci]]];
    uint32_t mask = 1u << ti;
    for (int e = lane; e < PAD; e += 32)
      for (int row = 0; row < S * n; ++row) Ci[row * RS + padc_s[e]] = 0.f;
    bool first = true;
    for (int64_t w0 = p_lo; w0 < p_hi || first; w0 += kWindow, first = false) {
      const int nwin = int(max(int64_t(0), min(int64_t(kWindow), p_hi - w0)));
      int count, start;
      __syncwarp();
      sort_window(a, w0, nwin, lane, count, start, [&](int slot, int64_t p, int s) {
        const double r = a.pair_dist[p];
        const SplinePos q = spline_pos(a.sp, r);
        // f_c RI = w.x y_k + w.y y''_k + w.z y_k+1 + w.w y''_k+1
        const float f = float(cutoff_fc(a, r)), fa = float(q.a), fb = float(q.b);
        wt[slot] = make_float4(f * fa, f * fa * (fa * fa - 1.f), f * fb, f * fb * (fb * fb - 1.f));
        geo[slot] = float(a.pair_dir[3 * p]);
        geo[kWindow + slot] = float(a.pair_dir[3 * p + 1]);
        geo[2 * kWindow + slot] = float(a.pair_dir[3 * p + 2]);
        gk[slot] = q.k;
        gs[slot] = s;
      });
      __syncwarp();
      mask |= __ballot_sync(0xffffffffu, count > 0);
      float acc[G][NV];
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[g][k] = 0.f;
      // the sums of species s are complete
      auto flush = [&](int s) {
        float * Cs = Ci + size_t(s) * n * RS;
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int k = 0; k < NV; ++k) {
            if (k < n && lane + 32 * g < K) {
              float * o = Cs + k * RS + col[g];
              float v = acc[g][k];
              // centre contribution (calculator_spherical_expansion.hh:2244-2247)
              if (first && s == ti && lane + 32 * g == 0) v += float(a.center_contrib[k]);
              *o = first ? v : *o + v;
            }
            acc[g][k] = 0.f;
          }
      };
      int s = 0;
      for (int at = 0; at < nwin; at += CH) {
        const int np = min(CH, nwin - at);
        if (hq < np) {
          float * y = Y + hq * SM::KP;
          pair_harmonics<L>(hc, geo[at + hq], geo[kWindow + at + hq], geo[2 * kWindow + at + hq], hj,
                            [&](int l, int m, float v, float re, float im) {
                              const int o = l * l + l;
                              if (m == 0) {
                                y[o] = v * 0.707106781186547524400844362104849039f;
                              } else {
                                y[o + m] = v * re;
                                y[o - m] = v * im;
                              }
                            });
        }
        for (int c = lane; c < W; c += 32) {
          float * o = R + dst_s[c];
          const float4 * col0 = a.sp.q4f + c;
#pragma unroll
          for (int q = 0; q < CH; ++q)
            if (q < np) {
              const float4 t = __ldg(col0 + size_t(gk[at + q]) * W), w = wt[at + q];
              o[q * SM::RI] = fmaf(w.w, t.w, fmaf(w.z, t.z, fmaf(w.y, t.y, w.x * t.x)));
            }
        }
        __syncwarp();
        for (int q = 0; q < np; ++q) {
          for (const int sq = gs[at + q]; s < sq; ++s) flush(s);
#pragma unroll
          for (int g = 0; g < G; ++g) {
            if (g + 1 == G && lane + 32 * g >= K) break;
            const float y = Y[q * SM::KP + lane + 32 * g];
            const float4 * r = reinterpret_cast<const float4 *>(R + q * SM::RI + lg[g]);
#pragma unroll
            for (int k = 0; k < NV / 4; ++k) {
              const float4 v = r[k];
              acc[g][4 * k] = fmaf(v.x, y, acc[g][4 * k]);
              acc[g][4 * k + 1] = fmaf(v.y, y, acc[g][4 * k + 1]);
              acc[g][4 * k + 2] = fmaf(v.z, y, acc[g][4 * k + 2]);
              acc[g][4 * k + 3] = fmaf(v.w, y, acc[g][4 * k + 3]);
            }
          }
        }
        __syncwarp();
      }
      for (; s < S; ++s) flush(s);
    }
    if (lane == 0) present[ci] = mask;
  }
}

// Few neighbours (see launch_expansion_fp32): the pairs of a centre in chunks
// of CH, each chunk's sums added to the coefficients in global memory:
//   (a) lanes = pairs: f_c, the spline interval and Y_lm of one pair each;
//   (b) lanes = radial channels: f_c RI_c(r_p) for the chunk's pairs one
//       after the other, one 16-byte load of the interval table per channel;
//   (c) lanes = (l, four columns m of the padded l-block, four radial
//       channels): 16 accumulators per lane; per pair of a species one
//       16-byte load of Y and four loads of f_c RI feed 16 products; the
//       sums are written once, as 16-byte stores, into the padded row
//       layout [S*n][row_stride(L)] (Y is zero in the padding columns, so
//       the padding of every l-block is written as zero).
template <int L, int CH>
__global__ void __launch_bounds__(kMaxWarps * 32)
expansion_few_kernel(ExpansionArgs a, float * __restrict__ C, uint32_t * __restrict__ present) {
  constexpr int K = (L + 1) * (L + 1);
  constexpr int L1 = L + 1;
  constexpr int RS = row_stride(L), OL = offp(L + 1), NG = OL / 4;
  constexpr int kChunkF = CH, kPadF = CH + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;  // centres per block
  const int W = a.fd.W, S = a.fd.S, n = a.fd.n;
  const int wpad = (W * kPadF + 3) & ~3;  // keeps Yp 16-byte aligned
  float * RIf = reinterpret_cast<float *>(smem_raw) + size_t(wid) * (wpad + CH * RS);  // [W][kPadF]
  float * Yp = RIf + wpad;  // [CH][RS]: Y_lm of each pair in the padded column layout
  __shared__ float pa_s[kMaxWarps][32], pb_s[kMaxWarps][32], fc_s[kMaxWarps][32];
  __shared__ int pk_s[kMaxWarps][32];
  __shared__ uint8_t order_s[kMaxWarps][32];
  __shared__ int16_t colk[K];  // padded column of lm: offp(l) + m
  __shared__ uint8_t grp_l[NG];
  for (int lm = threadIdx.x; lm < K; lm += blockDim.x) {
    int l = 0;
    while ((l + 1) * (l + 1) <= lm) ++l;
    colk[lm] = int16_t(offp_rt(l) + (lm - l * l));
  }
  for (int g = threadIdx.x; g < NG; g += blockDim.x) {
    int l = 0;
    while (4 * g >= offp_rt(l + 1)) ++l;
    grp_l[g] = uint8_t(l);
  }
  for (int e = lane; e < CH * RS; e += 32) Yp[e] = 0.f;  // padding columns stay zero
  __syncthreads();
  const int nblk = (n + 3) >> 2;  // blocks of four radial channels
  // where this lane's channels c, c + 32, .. of the table (in (l, n) order) go:
  // rows of the tile in (n, l) order, since the sums' lanes read one n at many
  // l (-1: no such channel). Worked out once: with the divisions in the loop
  // over pairs, 20 000 centres with 20 neighbours of one species took 1.03 ms
  // at n = 16, l = 12 instead of 0.71, and 0.43 instead of 0.36 at n = 12, l = 9.
  constexpr int NC = (L1 * 16 + 31) / 32;
  int dst[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const int c = lane + 32 * k;
    dst[k] = c < W ? (c % n * L1 + c / n) * kPadF : -1;
  }
  for (int64_t ci = int64_t(blockIdx.x) * nw + wid; ci < a.n_centers; ci += int64_t(gridDim.x) * nw) {
    float * Ci = C + size_t(ci) * S * n * RS;
    const int64_t p_lo = a.pair_off[ci] + 1, p_hi = a.pair_off[ci + 1];
    const int ti = a.species_lut[a.types[a.center_atom[ci]]];
    uint32_t mask_all = 1u << ti;
    // the columns after the last l-block
    for (int j = lane; j < S * n * (RS - OL); j += 32) {
      const int row = j / (RS - OL), c = OL + (j - row * (RS - OL));
      Ci[row * RS + c] = 0.f;
    }
    bool first = true;
    for (int64_t p0 = p_lo; p0 < p_hi || first; p0 += kChunkF) {
      const int np = int(max(int64_t(0), min(int64_t(kChunkF), p_hi - p0)));
      int my_sp = 31;
      if (lane < np) {
        const int64_t p = p0 + lane;
        const double r = a.pair_dist[p];
        my_sp = a.species_lut[a.types[a.pair_j[p]]];
        const SplinePos q = spline_pos(a.sp, r);
        pk_s[wid][lane] = q.k;
        pa_s[wid][lane] = float(q.a);
        pb_s[wid][lane] = float(q.b);
        fc_s[wid][lane] = float(cutoff_fc(a, r));
        const float dx = float(a.pair_dir[3 * p]), dy = float(a.pair_dir[3 * p + 1]),
                    dz = float(a.pair_dir[3 * p + 2]);
        float * yrow = Yp + lane * RS;
        spherical_harmonics<L, false, float>(dx, dy, dz, [&](int lm, float y, float, float, float) {
          yrow[colk[lm]] = y;
        });
      }
      // stable order of the chunk's pairs by species
      int before = 0;
      unsigned my_mask = 0;
      for (int s = 0; s < S; ++s) {
        unsigned m = __ballot_sync(0xffffffffu, my_sp == s);
        if (my_sp == s) my_mask = m;
        if (s < my_sp) before += __popc(m);
        if (m) mask_all |= 1u << s;
      }
      if (lane < np) order_s[wid][before + __popc(my_mask & lanemask_lt())] = uint8_t(lane);
      __syncwarp();
      // lanes = radial channels c, c + 32, ..; several pairs per step and no
      // branch between a step's table loads, so that they are in flight
      // together
      auto radial = [&](auto count) {
        constexpr int N = decltype(count)::value, kPairs = N > 4 ? 2 : 4;
#pragma unroll kPairs
        for (int q = 0; q < np; ++q) {
          const float fa = pa_s[wid][q], fb = pb_s[wid][q], f = fc_s[wid][q];
          const float ca = fa * fa - 1.f, cb = fb * fb - 1.f;
          const float4 * row = a.sp.q4f + size_t(pk_s[wid][q]) * W + lane;
#pragma unroll
          for (int k = 0; k < N; ++k)
            if (dst[k] >= 0) {
              const float4 t = __ldg(row + 32 * k);
              RIf[dst[k] + q] = f * (fa * (t.x + ca * t.y) + fb * (t.z + cb * t.w));
            }
        }
      };
      if (NC > 2 && W > 64)
        radial(std::integral_constant<int, NC>{});
      else
        radial(std::integral_constant<int, (NC < 2 ? NC : 2)>{});
      __syncwarp();
      int start = 0;
      for (int s = 0; s < S; ++s) {
        const int cnt = __popc(__ballot_sync(0xffffffffu, my_sp == s));
        if (cnt > 0 || first) {
          float * Cs = Ci + size_t(s) * n * RS;
          for (int t = lane; t < NG * nblk; t += 32) {
            const int g = t % NG, n0 = 4 * (t / NG);
            const int l = grp_l[g], col = 4 * g;
            const float * ri = RIf + (n0 * L1 + l) * kPadF;  // channel (n0 + k, l) at + k L1 kPadF
            float acc[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
              for (int e = 0; e < 4; ++e) acc[k][e] = 0.f;
            for (int q = 0; q < cnt; ++q) {
              const int pl = order_s[wid][start + q];
              const float4 y = *reinterpret_cast<const float4 *>(Yp + pl * RS + col);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if (n0 + k < n) {
                  const float rv = ri[k * L1 * kPadF + pl];
                  acc[k][0] += rv * y.x;
                  acc[k][1] += rv * y.y;
                  acc[k][2] += rv * y.z;
                  acc[k][3] += rv * y.w;
                }
              }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int nn = n0 + k;
              if (nn < n) {
                float4 * dst = reinterpret_cast<float4 *>(Cs + nn * RS + col);
                if (first) {
                  // centre contribution (calculator_spherical_expansion.hh:2244-2247)
                  if (s == ti && col == 0) acc[k][0] += float(a.center_contrib[nn]);
                  *dst = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
                } else {
                  float4 o = *dst;
                  o.x += acc[k][0];
                  o.y += acc[k][1];
                  o.z += acc[k][2];
                  o.w += acc[k][3];
                  *dst = o;
                }
              }
            }
          }
        }
        start += cnt;
      }
      __syncwarp();
      first = false;
    }
    if (lane == 0) present[ci] = mask_all;
    __syncwarp();
  }
}

// Few centres (see launch_expansion_fp32): a block of four warps per centre,
// its pairs up to `chunk` at a time (more than one chunk adds to the
// coefficients in global memory):
//   (a) threads = pairs: distance, direction, spline weights, and the pair's
//       place in the chunk's order by species;
//   (b) threads = (pair, two orders m): Y_lm (pairs_f32.cuh); warps = pairs,
//       lanes = radial channels: f_c RI, the table rows read whole;
//   (c) threads = (species, four columns m of an l-block, four radial
//       channels): per pair of the species two 16-byte loads from shared
//       memory feed 16 products; the sums are written once, as 16-byte stores
//       into the padded row layout [S*n][row_stride(L)] (Y is zero in the
//       padding columns, so the padding of every l-block is written as zero).
// A small system waits for one centre's chain of these steps, which four warps
// shorten (150 centres, 34 neighbours, n = 8, l = 6: 29 -> 12.7 us; 216 with 46,
// n = 12, l = 9: 69 -> 28); with many centres their barriers and idle lanes
// cost more.
constexpr int kBlockThreads = 128;
template <int L>
__global__ void __launch_bounds__(kBlockThreads)
expansion_block_kernel(ExpansionArgs a, float * __restrict__ C, uint32_t * __restrict__ present, int chunk) {
  using P = PairShape<L>;
  constexpr int L1 = P::L1, NL = P::NL, RS = row_stride(L), OL = offp(L + 1), NG = OL / 4;
  constexpr int kWarps = kBlockThreads / 32, kMaxChunk = kBlockThreads;
  extern __shared__ __align__(16) float smf[];
  __shared__ HarmonicConstants<L> hc;
  __shared__ float4 wt[kMaxChunk];                // the spline's weights of each pair's nodes
  __shared__ float geo[3][kMaxChunk];             // its direction
  __shared__ int gk[kMaxChunk];                   // its spline interval
  __shared__ int16_t dst_s[L1 * 16];              // channel (l, n) of the table -> place in a radial row
  __shared__ int16_t counts[kMaxSpecies][kWarps];  // pairs of each species by warp
  __shared__ int16_t first_s[kMaxSpecies + 1];    // first slot of each species
  __shared__ uint8_t grp_l[NG];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int W = a.fd.W, S = a.fd.S, n = a.fd.n, nb = (n + 3) >> 2;  // blocks of four radial channels
  const int RW = L1 * 4 * nb;
  float * Y = smf;              // [chunk][RS]: padded columns of each pair, by species
  float * R = smf + chunk * RS;  // [chunk][l][n rounded up to 4]
  hc.fill();
  for (int c = threadIdx.x; c < W; c += kBlockThreads) dst_s[c] = int16_t(c / n * 4 * nb + c % n);
  for (int g = threadIdx.x; g < NG; g += kBlockThreads) {
    int l = 0;
    while (4 * g >= offp_rt(l + 1)) ++l;
    grp_l[g] = uint8_t(l);
  }
  // padding columns of Y and channels past n stay zero
  for (int e = threadIdx.x; e < chunk * (RS + RW); e += kBlockThreads) smf[e] = 0.f;
  __syncthreads();
  const int tasks = NG * nb;
  for (int64_t ci = blockIdx.x; ci < a.n_centers; ci += gridDim.x) {
    float * Ci = C + size_t(ci) * S * n * RS;
    const int64_t p_lo = a.pair_off[ci] + 1, p_hi = a.pair_off[ci + 1];
    const int ti = a.species_lut[a.types[a.center_atom[ci]]];
    uint32_t mask = 1u << ti;
    // the columns after the last l-block
    for (int e = threadIdx.x; e < S * n * (RS - OL); e += kBlockThreads)
      Ci[e / (RS - OL) * RS + OL + e % (RS - OL)] = 0.f;
    bool first = true;
    for (int64_t p0 = p_lo; p0 < p_hi || first; p0 += chunk, first = false) {
      const int np = int(max(int64_t(0), min(int64_t(chunk), p_hi - p0)));
      const int64_t p = p0 + threadIdx.x;
      const bool own = int(threadIdx.x) < np;
      const int sp = own ? a.species_lut[a.types[a.pair_j[p]]] : -1;
      int rank = 0;  // among the warp's pairs of the same species
      for (int s = 0; s < S; ++s) {
        const unsigned m = __ballot_sync(0xffffffffu, sp == s);
        if (lane == s) counts[s][wid] = int16_t(__popc(m));
        if (sp == s) rank = __popc(m & lanemask_lt());
      }
      __syncthreads();
      if (wid == 0) {
        int mine = 0;
        if (lane < S)
          for (int w = 0; w < kWarps; ++w) mine += counts[lane][w];
        mask |= __ballot_sync(0xffffffffu, mine > 0);
        int upto = mine;
#pragma unroll
        for (int o = 1; o < kMaxSpecies; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += u;
        }
        if (lane < S) first_s[lane + 1] = int16_t(upto);
        if (lane == 0) first_s[0] = 0;
      }
      __syncthreads();
      if (own) {
        int slot = first_s[sp] + rank;
        for (int w = 0; w < wid; ++w) slot += counts[sp][w];
        const double r = a.pair_dist[p];
        const SplinePos q = spline_pos(a.sp, r);
        // f_c RI = w.x y_k + w.y y''_k + w.z y_k+1 + w.w y''_k+1
        const float f = float(cutoff_fc(a, r)), fa = float(q.a), fb = float(q.b);
        wt[slot] = make_float4(f * fa, f * fa * (fa * fa - 1.f), f * fb, f * fb * (fb * fb - 1.f));
        gk[slot] = q.k;
        for (int d = 0; d < 3; ++d) geo[d][slot] = float(a.pair_dir[3 * p + d]);
      }
      __syncthreads();
      for (int q = threadIdx.x / NL; q < np && threadIdx.x < kBlockThreads / NL * NL; q += kBlockThreads / NL) {
        float * y = Y + q * RS;
        pair_harmonics<L>(hc, geo[0][q], geo[1][q], geo[2][q], threadIdx.x % NL,
                          [&](int l, int m, float v, float re, float im) {
                            float * o = y + offp_rt(l) + l;
                            if (m == 0) {
                              *o = v * 0.707106781186547524400844362104849039f;
                            } else {
                              o[m] = v * re;
                              o[-m] = v * im;
                            }
                          });
      }
      for (int c = lane; c < W; c += 32) {
        float * o = R + dst_s[c];
        const float4 * table = a.sp.q4f + c;
#pragma unroll 4
        for (int q = wid; q < np; q += kWarps) {
          const float4 t = __ldg(table + size_t(gk[q]) * W), w = wt[q];
          o[q * RW] = fmaf(w.w, t.w, fmaf(w.z, t.z, fmaf(w.y, t.y, w.x * t.x)));
        }
      }
      __syncthreads();
      for (int t = threadIdx.x; t < S * tasks; t += kBlockThreads) {
        const int s = t / tasks, u = t - s * tasks, b = u / NG, g = u - b * NG;
        const int q0 = first_s[s], q1 = first_s[s + 1];
        if (q0 == q1 && !first) continue;
        const float * yp = Y + 4 * g;
        const float * rp = R + grp_l[g] * 4 * nb + 4 * b;
        float acc[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[k][e] = 0.f;
#pragma unroll 2
        for (int q = q0; q < q1; ++q) {
          const float4 y = *reinterpret_cast<const float4 *>(yp + q * RS);
          const float4 r = *reinterpret_cast<const float4 *>(rp + q * RW);
          const float rv[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            acc[k][0] = fmaf(rv[k], y.x, acc[k][0]);
            acc[k][1] = fmaf(rv[k], y.y, acc[k][1]);
            acc[k][2] = fmaf(rv[k], y.z, acc[k][2]);
            acc[k][3] = fmaf(rv[k], y.w, acc[k][3]);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int nn = 4 * b + k;
          if (nn < n) {
            float4 * o = reinterpret_cast<float4 *>(Ci + (s * n + nn) * RS + 4 * g);
            float4 v = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
            if (first) {
              // centre contribution (calculator_spherical_expansion.hh:2244-2247)
              if (s == ti && g == 0) v.x += float(a.center_contrib[nn]);
            } else {
              const float4 before = *o;
              v = make_float4(before.x + v.x, before.y + v.y, before.z + v.z, before.w + v.w);
            }
            *o = v;
          }
        }
      }
      __syncthreads();  // Y, R and the counts are read no more
    }
    if (threadIdx.x == 0) present[ci] = mask;
  }
}

template <int L, int NV>
void launch_nv(const ExpansionArgs & a, float * C, uint32_t * present, cudaStream_t st) {
  const TileConfig cfg = tile_config(a.fd.S, a.fd.n, a.fd.L);
  const size_t per_warp = ExpSmem<L, NV>::kFloats * sizeof(float);
  const int warps = std::min(cfg.exp_warps, kMaxWarps);
  const size_t smem = warps * per_warp;
  auto kernel = expansion_f32_kernel<L, NV>;
  RGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  int dev = 0, sms = 148, per_sm = 1;
  RGPU_CUDA(cudaGetDevice(&dev));
  RGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  RGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem));
  const int64_t blocks = (a.n_centers + warps - 1) / warps;
  const int grid = int(std::min<int64_t>(blocks, int64_t(sms) * std::max(per_sm, 1) * 4));
  kernel<<<grid, warps * 32, smem, st>>>(a, C, present);
}

void launch_few(const ExpansionArgs & a, float * C, uint32_t * present, cudaStream_t st) {
  const TileConfig cfg = tile_config(a.fd.S, a.fd.n, a.fd.L);
  const int CH = cfg.exp_chunk;
  int dev = 0, sms = 148, optin = 0;
  RGPU_CUDA(cudaGetDevice(&dev));
  RGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  RGPU_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t per_warp =
      ((size_t(a.fd.W) * (CH + 1) + 3) / 4 * 4 + size_t(CH) * row_stride(a.fd.L)) * sizeof(float);
  const int warps = int(std::max<size_t>(1, std::min<size_t>(size_t(cfg.exp_warps), (size_t(optin) - 8192) / per_warp)));
  const size_t smem = size_t(warps) * per_warp;
  int grid = int(std::min<int64_t>((a.n_centers + warps - 1) / warps, int64_t(sms) * 16 * (4 / std::min(warps, 4))));
#define RGPU_EXPF_NV(LL, CHH)                                                                       \
  {                                                                                                 \
    RGPU_CUDA(cudaFuncSetAttribute(expansion_few_kernel<LL, CHH>,                                   \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));        \
    expansion_few_kernel<LL, CHH><<<grid, warps * 32, smem, st>>>(a, C, present);                   \
  }
#define RGPU_EXP_CASE(LL)              \
  case LL:                             \
    if (CH == 8) {                     \
      RGPU_EXPF_NV(LL, 8)              \
    } else if (CH == 32) {             \
      RGPU_EXPF_NV(LL, 32)             \
    } else {                           \
      RGPU_EXPF_NV(LL, 16)             \
    }                                  \
    break;
  switch (a.fd.L) {
    RGPU_EXP_CASE(0)
    RGPU_EXP_CASE(1)
    RGPU_EXP_CASE(2)
    RGPU_EXP_CASE(3)
    RGPU_EXP_CASE(4)
    RGPU_EXP_CASE(5)
    RGPU_EXP_CASE(6)
    RGPU_EXP_CASE(7)
    RGPU_EXP_CASE(8)
    RGPU_EXP_CASE(9)
    RGPU_EXP_CASE(10)
    RGPU_EXP_CASE(11)
    RGPU_EXP_CASE(12)
    default:
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_angular above 12 is not supported on the GPU");
  }
#undef RGPU_EXP_CASE
#undef RGPU_EXPF_NV
}

template <int L>
void launch_block(const ExpansionArgs & a, float * C, uint32_t * present, cudaStream_t st) {
  const size_t per_pair = (row_stride(L) + size_t(L + 1) * ((a.fd.n + 3) / 4 * 4)) * sizeof(float);
  // pairs at a time: a warp's number on each of the four, while five blocks fit on an SM
  int chunk = 4 * tile_config(a.fd.S, a.fd.n, a.fd.L).exp_chunk;
  while (chunk > 16 && chunk * per_pair > 44 * 1024) chunk /= 2;
  const size_t smem = chunk * per_pair;
  auto kernel = expansion_block_kernel<L>;
  RGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  int dev = 0, sms = 148, per_sm = 1;
  RGPU_CUDA(cudaGetDevice(&dev));
  RGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  RGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlockThreads, smem));
  const int grid = int(std::min<int64_t>(a.n_centers, int64_t(sms) * std::max(per_sm, 1) * 4));
  kernel<<<grid, kBlockThreads, smem, st>>>(a, C, present, chunk);
}

}  // namespace

void launch_expansion_fp32(const ExpansionArgs & a, float * C, uint32_t * present, cudaStream_t st) {
  if (a.n_centers == 0) return;
  if (a.fd.n > 16) throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_radial above 16 is not supported on the fast path");
  sph_constants_tu();
  int dev = 0, sms = 148;
  RGPU_CUDA(cudaGetDevice(&dev));
  RGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const bool block = a.n_centers <= kFewCentres * sms;
  const int sums = (a.fd.K + 31) / 32 * (a.fd.n <= 8 ? 8 : a.fd.n <= 12 ? 12 : 16);
  const bool few = a.n_pairs < kFewPairs * a.n_centers || (a.fd.S == 1 && (sums <= kSumsLow || sums >= kSumsHigh));
  if (!block && few) {
    launch_few(a, C, present, st);
    RGPU_LAUNCHED();
    RGPU_CUDA(cudaGetLastError());
    return;
  }
#define RGPU_CASE(LL)                            \
  case LL:                                       \
    if (block)                                   \
      launch_block<LL>(a, C, present, st);       \
    else if (a.fd.n <= 8)                        \
      launch_nv<LL, 8>(a, C, present, st);       \
    else if (a.fd.n <= 12)                       \
      launch_nv<LL, 12>(a, C, present, st);      \
    else                                         \
      launch_nv<LL, 16>(a, C, present, st);      \
    break;
  switch (a.fd.L) {
    RGPU_CASE(0)
    RGPU_CASE(1)
    RGPU_CASE(2)
    RGPU_CASE(3)
    RGPU_CASE(4)
    RGPU_CASE(5)
    RGPU_CASE(6)
    RGPU_CASE(7)
    RGPU_CASE(8)
    RGPU_CASE(9)
    RGPU_CASE(10)
    RGPU_CASE(11)
    RGPU_CASE(12)
    default:
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_angular above 12 is not supported on the GPU");
  }
#undef RGPU_CASE
  RGPU_LAUNCHED();
  RGPU_CUDA(cudaGetLastError());
}

}  // namespace rgpu
