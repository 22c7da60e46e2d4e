// gemm_fp64.cuh -- the grouped FP64 product tiles shared by the forward
// commutator (kernels_comm.cu) and its adjoint (adjoint.cu).
//
// What bounds them: the FP64 pipe.  GB300 retires about two FP64 FMAs per SM
// and cycle (one warp instruction per 16 cycles), so an operand load per FMA
// costs next to nothing and the time is the number of warp FMAs issued, padding
// included, over the SMs' even shares.  So there is no shared-memory staging
// (a warp streams its operands from L1/L2, its next four k in flight), and the
// tile follows the live outputs instead: a warp owns 16 x 16 outputs, lanes 8 x
// 4, and issues only the 8-row and 4-column groups that hold some.  A CTA is
// four such warps, side by side (32 x 32 outputs) or, where one warp's
// contraction would be a large part of an SM's share of the whole list, on one
// 16 x 16 output with a quarter of K each, added in warp order through shared
// memory.  Tiles run longest first.
//
// Measured on one GPU against 64 x 64 shared-memory tiles of 256 threads: FP64
// commutators 703 -> 494 us at emax = 6 (padding 4 % instead of 25 %) and 115 ->
// 40 us at emax = 4; adjoints 1430 -> 850 us and 272 -> 119 us.
#pragma once

#include <algorithm>

#include "device.cuh"

namespace imsrg {

constexpr int GT_THREADS = 128;
// CTAs per SM: 16 warps hide the operand loads.  At its 128 registers a build spills
// 4 bytes of stores and 32 of loads in the plain and the adjoint's kernel, none in
// the merged one; five or six spill more and are slower.
constexpr int GT_CTAS = 4;

// Host side: tiles of problems with outputs m x n and contraction work k (the
// sum of the terms' lengths), longest first.  split[p]: see gemm_split.
struct GemmShape {
  int m, n;
  long k;
  int split;
};

// Whether problem p splits K over the CTA's warps: a warp's serial FMAs (8 per
// k) would exceed `share` of one warp scheduler's part of all the work.  The
// line: with few tiles (small bases) the longest warp is the kernel's time, with
// many the split's extra additions cost more than the shorter tail gives.  A
// tenth: emax 4 / 6 commutators 38.4 / 491 us and adjoints 117 / 831 us; never
// splitting 52 / 488 and 130 / 889, always splitting 40 / 700 and 117 / 955.
inline void gemm_split(std::vector<GemmShape> &ps, int num_sms) {
  constexpr double share = 0.1;
  double total = 0.0;
  for (const GemmShape &p : ps) total += (double)((p.m + 7) / 8) * ((p.n + 3) / 4) * p.k;
  const double part = total / (4.0 * num_sms);
  for (GemmShape &p : ps) p.split = 8.0 * p.k > share * part && p.k >= 8;
}

inline std::vector<GemmTile> gemm_tiles(const std::vector<GemmShape> &ps) {
  std::vector<GemmTile> t;
  std::vector<std::pair<long, int>> order;
  for (int p = 0; p < (int)ps.size(); p++) {
    const int w = ps[p].split ? 16 : 32;
    for (int n0 = 0; n0 < ps[p].n; n0 += w)
      for (int m0 = 0; m0 < ps[p].m; m0 += w) {
        const long rows = std::min(16, ps[p].m - m0), cols = std::min(16, ps[p].n - n0);
        order.push_back({-((rows + 7) / 8) * ((cols + 3) / 4) * ps[p].k / (ps[p].split ? 4 : 1), (int)t.size()});
        t.push_back({p, m0, n0, ps[p].split});
      }
  }
  std::stable_sort(order.begin(), order.end(),
                   [](const std::pair<long, int> &a, const std::pair<long, int> &b) { return a.first < b.first; });
  std::vector<GemmTile> out;
  for (const std::pair<long, int> &o : order) out.push_back(t[o.second]);
  return out;
}

// part(i, j) += (-1)^neg sum over k in [k0, k1) of A(m, k) B(k, n) for the rows m =
// m0 + r + 8 i and columns n = n0 + c + 4 j of lane (r, c); element (m, k) of A at
// m sam + k sak, (k, n) of B at k sbk + n sbn.  Rows past M and columns past N
// repeat the last one (their sums are not stored).  Ascending k: each sum's
// rounding does not depend on the tile.  The sign flips A on the integer pipe.
template <int NI, int NJ>
__device__ __forceinline__ void gemm_mac(const double *A, long sam, long sak, const double *B, long sbk, long sbn,
                                         int M, int N, int m0, int n0, int k0, int k1, int neg,
                                         double (&part)[NI][NJ]) {
  constexpr int KU = 2;  // k per load group: 1 leaves loads exposed (705 us at emax = 6), 4 takes 206 registers (523 us)
  const int r = threadIdx.x & 7, c = (threadIdx.x >> 3) & 3;
  const double *pa[NI], *pb[NJ];
#pragma unroll
  for (int i = 0; i < NI; i++) pa[i] = A + min(m0 + r + 8 * i, M - 1) * sam + k0 * sak;
#pragma unroll
  for (int j = 0; j < NJ; j++) pb[j] = B + min(n0 + c + 4 * j, N - 1) * sbn + k0 * sbk;
  double a[KU][NI], b[KU][NJ];
  auto load = [&](int k) {  // k .. k + KU - 1, those below k1
#pragma unroll
    for (int u = 0; u < KU; u++)
      if (k + u < k1) {
#pragma unroll
        for (int i = 0; i < NI; i++) a[u][i] = pa[i][u * sak];
#pragma unroll
        for (int j = 0; j < NJ; j++) b[u][j] = pb[j][u * sbk];
      }
#pragma unroll
    for (int i = 0; i < NI; i++) pa[i] += KU * sak;
#pragma unroll
    for (int j = 0; j < NJ; j++) pb[j] += KU * sbk;
  };
  load(k0);
  for (int k = k0; k < k1; k += KU) {
    double x[KU][NI], y[KU][NJ];
#pragma unroll
    for (int u = 0; u < KU; u++) {
#pragma unroll
      for (int i = 0; i < NI; i++) x[u][i] = dflip(a[u][i], neg);
#pragma unroll
      for (int j = 0; j < NJ; j++) y[u][j] = b[u][j];
    }
    if (k + KU < k1) load(k + KU);
#pragma unroll
    for (int u = 0; u < KU; u++)
      if (k + u < k1) {
#pragma unroll
        for (int i = 0; i < NI; i++)
#pragma unroll
          for (int j = 0; j < NJ; j++) part[i][j] = fma(x[u][i], y[u][j], part[i][j]);
      }
  }
}

// One warp's outputs: `terms(it, add)` calls add(A, sam, sak, B, sbk, sbn, K,
// neg) for term it; C(m, n) at C[m + n ldc] is set, or added to (ADD).
template <int NI, int NJ, bool ADD, typename Terms>
__device__ __forceinline__ void gemm_warp_tile(const Terms &terms, int nterms, int M, int N, int m0, int n0, int split,
                                               int w, double *C, int ldc, double (*red)[256]) {
  double acc[NI][NJ];
#pragma unroll
  for (int i = 0; i < NI; i++)
#pragma unroll
    for (int j = 0; j < NJ; j++) acc[i][j] = 0.0;
  for (int it = 0; it < nterms; it++)
    terms(it, [&](const double *A, long sam, long sak, const double *B, long sbk, long sbn, int K, int neg) {
      const int k0 = split ? (int)((long)K * w / 4) : 0, k1 = split ? (int)((long)K * (w + 1) / 4) : K;
      if (k0 >= k1) return;
      double part[NI][NJ];
#pragma unroll
      for (int i = 0; i < NI; i++)
#pragma unroll
        for (int j = 0; j < NJ; j++) part[i][j] = 0.0;
      gemm_mac<NI, NJ>(A, sam, sak, B, sbk, sbn, M, N, m0, n0, k0, k1, neg, part);
      // each term's sum by itself; the first one costs no addition
#pragma unroll
      for (int i = 0; i < NI; i++)
#pragma unroll
        for (int j = 0; j < NJ; j++) {
          if (it == 0) acc[i][j] = part[i][j];
          else acc[i][j] += part[i][j];
        }
    });
  const int lane = threadIdx.x & 31, r = lane & 7, c = lane >> 3;
  if (split) {  // the quarters of K in warp order (block-uniform)
#pragma unroll
    for (int i = 0; i < NI; i++)
#pragma unroll
      for (int j = 0; j < NJ; j++)
        if (w > 0) red[w - 1][(i * NJ + j) * 32 + lane] = acc[i][j];
    __syncthreads();
    if (w > 0) return;
#pragma unroll
    for (int i = 0; i < NI; i++)
#pragma unroll
      for (int j = 0; j < NJ; j++)
        acc[i][j] = ((acc[i][j] + red[0][(i * NJ + j) * 32 + lane]) + red[1][(i * NJ + j) * 32 + lane]) +
                    red[2][(i * NJ + j) * 32 + lane];
  }
#pragma unroll
  for (int j = 0; j < NJ; j++) {
    const int n = n0 + c + 4 * j;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int m = m0 + r + 8 * i;
      if (m < M && n < N) {
        double *p = C + m + (long)n * ldc;
        *p = ADD ? *p + acc[i][j] : acc[i][j];
      }
    }
  }
}

// One CTA's tile.  The warps of an unsplit tile rotate over its quadrants with
// the CTA index, so ragged edges do not always idle the same warp scheduler.
template <bool ADD, typename Terms>
__device__ __forceinline__ void gemm_cta_tile(const GemmTile &t, const Terms &terms, int nterms, int M, int N,
                                              double *C, int ldc) {
  __shared__ double red[3][256];
  const int w = ((threadIdx.x >> 5) + (t.split ? 0 : blockIdx.x)) & 3;
  const int m0 = t.m0 + (t.split ? 0 : 16 * (w & 1)), n0 = t.n0 + (t.split ? 0 : 16 * (w >> 1));
  if (m0 >= M || n0 >= N) return;  // never in a split tile
  const int ni = M - m0 > 8 ? 2 : 1, nj = min(4, (N - n0 + 3) >> 2);
#define GEMM_CASE(I, J) \
  case (I - 1) * 4 + J - 1: gemm_warp_tile<I, J, ADD>(terms, nterms, M, N, m0, n0, t.split, w, C, ldc, red); break;
  switch ((ni - 1) * 4 + nj - 1) {
    GEMM_CASE(1, 1)
    GEMM_CASE(1, 2)
    GEMM_CASE(1, 3)
    GEMM_CASE(1, 4)
    GEMM_CASE(2, 1)
    GEMM_CASE(2, 2)
    GEMM_CASE(2, 3)
    GEMM_CASE(2, 4)
  }
#undef GEMM_CASE
}

}  // namespace imsrg
