// What the FP32 expansion kernels share:
//   * harmonics (lanes = (pair, two orders m)): each lane runs the recursions
//     in l of the orders m = j and m = L - j, L + 2 steps together whatever j,
//     so a warp evaluates 32 / ceil((L + 1) / 2) pairs (8 at L = 6) at once
//     with few lanes idle; one lane per pair left 24 of 32 idle for the eight
//     pairs a centre and species has at a time;
//   * the order of a centre's pairs by neighbour species, a window at a time.
#pragma once

#include "common.cuh"

namespace rgpu {

constexpr int kWindow = 96;  // pairs sorted at a time (a centre with more takes several windows)

template <int L>
struct PairShape {
  static constexpr int L1 = L + 1, K = L1 * L1;
  static constexpr int NL = (L + 2) / 2;                          // lanes per pair in the harmonics
  static constexpr int CH = 32 / NL < 8 ? 32 / NL : 8;            // pairs per chunk
  static constexpr int G = (K + 31) / 32;                         // lane groups over lm
};

// Recursion constants of the harmonics in shared memory (per block):
// P_lm / sin^m = q_lm with q_mm = cmm[m], q_lm = rec.x z q_(l-1)m + rec.y
// q_(l-2)m, the factors of math/spherical_harmonics.cc:54-71.
template <int L>
struct HarmonicConstants {
  float2 rec[(L + 1) * (L + 1)];  // [m][l], l > m
  float cmm[L + 1];
  __device__ void fill() {
    constexpr int S = kMaxL + 2;
    for (int e = threadIdx.x; e < (L + 1) * (L + 1); e += blockDim.x) {
      const int m = e / (L + 1), l = e - m * (L + 1);
      float2 r = make_float2(0.f, 0.f);
      if (l == m + 1) r.x = SphC<float>::c1(l);
      if (l > m + 1) r = make_float2(SphC<float>::a(l * S + m), SphC<float>::a(l * S + m) * SphC<float>::b(l * S + m));
      rec[e] = r;
    }
    for (int m = threadIdx.x; m <= L; m += blockDim.x) {
      float v = 0.398942280401432677939946059934381868f;  // sqrt(1/(2 pi))
      for (int k = 1; k <= m; ++k) v *= SphC<float>::c2(k);
      cmm[m] = v;
    }
  }
};

// The harmonics of the unit vector (x, y, z) that belong to lane j of the
// pair's NL lanes. emit(l, m, q, re, im) gets, for every l >= m of its orders,
// q_lm and (x + iy)^m: Y_l,m = q re, Y_l,-m = q im (m > 0), Y_l0 = q / sqrt2.
template <int L, class Emit>
__device__ __forceinline__ void pair_harmonics(const HarmonicConstants<L> & c, float x, float y, float z, int j,
                                               Emit && emit) {
  const int m2 = L - j;
  float re = 1.f, im = 0.f;
  float ra = 1.f, ia = 0.f;  // power j
  float rb = 1.f, ib = 0.f;  // power L - j
#pragma unroll
  for (int k = 1; k <= L; ++k) {
    const float nr = re * x - im * y, ni = re * y + im * x;
    if (k == j) ra = nr, ia = ni;
    if (k == m2) rb = nr, ib = ni;
    re = nr;
    im = ni;
  }
  int m = j, l = j;
  bool on = true;
  float q0 = c.cmm[j], q1 = 0.f;
#pragma unroll
  for (int step = 0; step < L + 2; ++step) {
    if (on) emit(l, m, q0, ra, ia);
    if (l < L) {
      ++l;
      const float2 r = c.rec[m * (L + 1) + l];
      const float q = r.x * z * q0 + r.y * q1;
      q1 = q0;
      q0 = q;
    } else {
      on = m < m2;  // the second order, once
      m = l = m2;
      q0 = c.cmm[m2];
      q1 = 0.f;
      ra = rb, ia = ib;
    }
  }
}

// The pairs [p0, p0 + n) (n <= kWindow) sorted by neighbour species: put(slot,
// p, species) is called for each, slot its place in that (stable) order. Lane
// s gets the number of pairs of species s in `count` and their first slot in
// `start`.
template <class Put>
__device__ __forceinline__ void sort_window(const ExpansionArgs & a, int64_t p0, int n, int lane, int & count,
                                            int & start, Put && put) {
  int sp[kWindow / 32];
  count = 0;
#pragma unroll
  for (int b = 0; b < kWindow / 32; ++b) {
    const int i = 32 * b + lane;
    sp[b] = i < n ? a.species_lut[a.types[a.pair_j[p0 + i]]] : -1;
    if (32 * b < n)
      for (int s = 0; s < a.fd.S; ++s) {
        const unsigned m = __ballot_sync(0xffffffffu, sp[b] == s);
        if (lane == s) count += __popc(m);
      }
  }
  int x = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  start = x - count;
  int cursor = start;
#pragma unroll
  for (int b = 0; b < kWindow / 32; ++b) {
    if (32 * b >= n) break;
    int slot = -1;
    for (int s = 0; s < a.fd.S; ++s) {
      const unsigned m = __ballot_sync(0xffffffffu, sp[b] == s);
      const int at = __shfl_sync(0xffffffffu, cursor, s);
      if (sp[b] == s) slot = at + __popc(m & lanemask_lt());
      if (lane == s) cursor += __popc(m);
    }
    if (slot >= 0) put(slot, p0 + 32 * b + lane, sp[b]);
  }
}

}  // namespace rgpu
