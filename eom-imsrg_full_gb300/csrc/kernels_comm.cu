// kernels_comm.cu -- FP64 kernels of one scalar-scalar commutator [L, R].
//
// One commutator is these launches:
//   1. front           Pandya transform of L and R into LCC, RCC
//                      (calculate_cross_coupled, cross_coupled.f90:1190-1300),
//                      and in split precision the block exponents
//   2. sums_122        commutator_122 of every two-body element (commutators.f90:
//                      283-396), which needs only L and R (front.cuh)
//   3. gemm_fp64       every dense contraction as one grouped GEMM: the 12
//                      ladder products per (2J,Tz,parity) block of
//                      commutator_222_pp_hh (commutators.f90:596-766) and the
//                      WCC = LCC RCC^T products of commutator_222_ph (:792-802)
//                      (the split-precision path has its slicing and tensor-core
//                      launches instead)
//   4. ph_inputs +     every two-body element of RES: the antisymmetrised ladder
//      assemble_2body  epilogue of 222_pp_hh (:658-764) and the inverse Pandya
//                      recoupling of 222_ph (:804-923) on top of the 122 sums
//   5. one_body        every one-body element: commutator_111 (:36-80),
//                      121 (:83-280) and 221 (:435-578) (front.cuh)
//   6. e0              E0 from 110 + 220 (:10-33, :399-432), which need only
//                      L and R
// 1, 3 and 4 follow one another on the basis stream; the others run on side
// streams beside them, or in split precision on small bases inside their
// launches (commutator_launches).
// No float atomics: every reduction has a fixed order, so results are
// bit-reproducible run to run.
#include "front.cuh"
#include "gemm_fp64.cuh"

namespace imsrg {

namespace {

// ---------------------------------------------------------------------------
// 1. Pandya transform: CCX(r(a,b), nb(p,h)) of cross_coupled.f90:1247-1291.
// ---------------------------------------------------------------------------
// exps != nullptr (split-precision path, ccf_packed): also the largest IEEE
// exponent of every LCC block (into exps[gL + block]) and RCC block (exps[gR +
// block]) for the digit slicing: lanes of a warp that share a block combine
// theirs, one integer atomicMax per block and warp (order-independent).
// SIDES: 1 = LCC only, 2 = RCC only, 3 = both from one pass over the gather
// list (the separate passes let the RCC half run while L is still arriving).
template <int SIDES>
__device__ __forceinline__ void cc_forward(const DevTables &T, const double *__restrict__ L, int hL,
                                           const double *__restrict__ R, int hR, double *LCC, double *RCC, int *exps,
                                           int gL, int gR, int cta) {
  const long t = (long)cta * blockDim.x + threadIdx.x;
  int q1 = -1, xL = 0, xR = 0;
  if (t < T.cc_total) {
    const int v = T.ccf_order[t];  // elements grouped by term count
    const long e = T.ccf_packed ? (v & 0xFFFFFF) : v;
    if (T.ccf_packed) q1 = v >> 24;
    const int k0 = T.cct_start[e], k1 = T.cct_start[e + 1];
    const int nL = hL < 0, nR = hR < 0;
    double sl = 0.0, sr = 0.0;
    for (int k = k0; k < k1; k++) {
      const int ix = T.cct_idx[k];
      const int tr = (int)((unsigned)ix >> 31), idx = ix & 0x7fffffff;
      const double c = T.cct_coef[k];
      if (SIDES & 1) sl = fma(c, dflip(L[idx], tr & nL), sl);
      if (SIDES & 2) sr = fma(c, dflip(R[idx], tr & nR), sr);
    }
    if (SIDES & 1) {
      LCC[e] = sl;
      xL = (int)((__double_as_longlong(sl) >> 52) & 0x7FF);
    }
    if (SIDES & 2) {
      RCC[e] = sr;
      xR = (int)((__double_as_longlong(sr) >> 52) & 0x7FF);
    }
  }
  if (exps) {  // every lane of the warp takes part (no early exit above)
    const unsigned peers = __match_any_sync(0xffffffffu, q1);
    const int mL = __reduce_max_sync(peers, xL), mR = __reduce_max_sync(peers, xR);
    if (q1 >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) {
      if (SIDES & 1) atomicMax(exps + gL + q1, mL);
      if (SIDES & 2) atomicMax(exps + gR + q1, mR);
    }
  }
}

constexpr int CC_THREADS = 256;

// Largest biased exponent of one chunk (at most kOzChunk elements) of an exponent
// group into out[group]: integer atomicMax, order-independent, so deterministic.
__device__ __forceinline__ void exponents(const OzChunk &c, const double *L, const double *R, const double *LCC,
                                          const double *RCC, int *out) {
  __shared__ int sh[CC_THREADS / 32];
  const double *src = (c.src == 0 ? L : c.src == 1 ? R : c.src == 2 ? LCC : RCC) + c.off;
  int m = 0;
#pragma unroll
  for (int k = 0; k < kOzChunk / CC_THREADS; k++) {  // independent loads
    const int i = threadIdx.x + k * CC_THREADS;
    if (i < c.len) m = max(m, (int)((__double_as_longlong(src[i]) >> 52) & 0x7FF));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < CC_THREADS / 32; w++) m = max(m, sh[w]);
    atomicMax(&out[c.group], m);
  }
}

// CTAs [0, nexp): exponent chunks; the rest: the Pandya transform.
struct FrontArgs {
  const OzChunk *chunks;
  int *exps;  // of the chunks
  int nexp;
};
template <int SIDES>
__global__ void __launch_bounds__(CC_THREADS) k_front(DevTables T, const double *__restrict__ L, int hL,
                                                      const double *__restrict__ R, int hR, double *LCC, double *RCC,
                                                      int *exps, int gL, int gR, FrontArgs f) {
  pdl_go();
  const int cta = blockIdx.x;
  if (cta < f.nexp) exponents(f.chunks[cta], L, R, LCC, RCC, f.exps);
  else if (SIDES) cc_forward<SIDES>(T, L, hL, R, hR, LCC, RCC, exps, gL, gR, cta - f.nexp);
}

// The 122 sums alone (40 registers: beside the one-body part's 54 they took the
// slicing's and the products' share of an SM, emax 6 104.8 us -> 108.4).
__global__ void __launch_bounds__(FRONT_THREADS) k_sums_122(DevTables T, SumsArgs a) {
  sums_122(T, a, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// 2. Grouped FP64 products: C = sum_t alpha_t op(A_t) op(B_t), one CTA per tile
//    of the list (gemm_fp64.cuh).  ABS: a merged list of several bases (absolute
//    pointers, tiles of bases with act[inst] == 0 skipped).
// ---------------------------------------------------------------------------
template <bool ABS>
__global__ void __launch_bounds__(GT_THREADS, GT_CTAS) k_gemm_fp64(const GemmProb *__restrict__ probs,
                                                          const GemmTile *__restrict__ tiles, Operands ops, int hL,
                                                          int hR, const int *__restrict__ act) {
  const GemmTile t = tiles[blockIdx.x];
  const GemmProb &P = probs[t.prob];
  pdl_go();
  pdl_wait();
  if (ABS && act && !act[P.inst]) return;  // block-uniform
  double *C = ABS ? P.c_abs : ops.dst[P.c_dst] + P.c_off;
  gemm_cta_tile<false>(
      t,
      [&](int it, auto add) {
        const GemmTerm &m = P.t[it];
        const double *A = ABS ? m.a_abs : ops.src[m.a_src] + m.a_off;
        const double *B = ABS ? m.b_abs : ops.src[m.b_src] + m.b_off;
        add(A, m.ta ? (long)m.lda : 1L, m.ta ? 1L : (long)m.lda, B, m.tb ? (long)m.ldb : 1L, m.tb ? 1L : (long)m.ldb,
            P.K, (m.coef < 0) ^ (m.use_hl && hL < 0) ^ (m.use_hr && hR < 0));  // coefficients are +-1
      },
      P.nterms, P.M, P.N, C, P.ldc);
}

// ---------------------------------------------------------------------------
// 3. Two-body assembly from the per-element gather lists (see Asm2Head).
// ---------------------------------------------------------------------------
// Z from its four entries (see PhPatch): FP64, or the split engine's exact int64
// level sums (WCC = v 2^k), combined exactly before one conversion.
template <bool INT>
__device__ __forceinline__ double ph_combine(double w1, double w2, double w3, double w4, int nph, int hL, int hR,
                                             int k) {
  if (!INT) {
    const double a = w1 + dflip(w2, nph), c = dflip(w3, nph) + w4;
    return dflip(a, hL < 0) - dflip(c, hR < 0);
  }
  const long long i2 = __double_as_longlong(w2), i3 = __double_as_longlong(w3);
  const long long a = __double_as_longlong(w1) + (nph ? -i2 : i2);
  const long long c = (nph ? -i3 : i3) + __double_as_longlong(w4);
  const long long z = (hL < 0 ? -a : a) - (hR < 0 ? -c : c);
  // z 2^k: add k to the exponent field on the integer pipe when the result
  // stays normal (exactly ldexp's value), else ldexp
  double d = (double)z;
  unsigned long long bits = (unsigned long long)__double_as_longlong(d);
  const int E = (int)((bits >> 52) & 0x7FF);
  if (E != 0 && E + k > 0 && E + k < 2047) {
    bits += (unsigned long long)(long long)k << 52;
    d = __longlong_as_double((long long)bits);
  } else if (E != 0) {
    d = ldexp(d, k);
  }
  return d;
}

// Recoupling inputs Z of commutator_222_ph, large bases: four CTAs per 32 x 32
// patch of a block's (x, y) plane, an input per thread (see PhPatch).  W(x, y)
// and W(x', y') are read along their columns; W(y, x) and W(y', x') across
// theirs, the CTA's eight rows sharing sectors; each value goes to its place in
// Z.  What bounds it: the latency of the reads, now independent of one another
// once the patch is known, and then their sectors (3.5 million at emax = 6
// against 6.3 million of one thread per input in the order of Z).
template <bool INT>
__global__ void __launch_bounds__(256) k_ph_patches(DevTables T, const double *WCC, int hL, int hR,
                                                    const int *exps, int gL, int gR, int kshift, double *Z) {
  const PhPatch &p = T.ph_patch[blockIdx.x >> 2];
  const int layers = p.layers;
  const int lane = threadIdx.x & 31, ty = (threadIdx.x >> 5) + (blockIdx.x & 3) * 8, rl = p.rlen;
  pdl_go();
  pdl_wait();
  if (layers == 0) return;
  const double *W = WCC + p.w, *V = WCC + p.v;
  const unsigned *slots = T.ph_slots + (long)p.table * 1024 + ty * 32 + lane;
  const unsigned char *ph = T.cc_rowph + p.row0;
  const int x = p.x0 + lane, y = p.y0 + ty;
  if (x >= rl || y >= rl) return;
  const int xr = ph_rev(p, x), yr = ph_rev(p, y);
  unsigned u = __ldg(slots);
  const double w1 = W[x + (long)y * rl], w2 = V[yr + (long)xr * rl], w3 = V[xr + (long)yr * rl],
               w4 = W[y + (long)x * rl];
  const int nph = __ldg(ph + x) ^ __ldg(ph + y);
  const int k = INT ? (exps[gL + p.group] - 1022) + (exps[gR + p.group] - 1022) - kshift : 0;
  const double d = ph_combine<INT>(w1, w2, w3, w4, nph, hL, hR, k);
  for (int l = 0;;) {
    if ((u & kPhSlot) != kPhNone) Z[u & kPhSlot] = dflip(d, ((u & kPhFlip) != 0) ^ ((u & kPhSwap) && hL * hR > 0));
    if (++l == layers) break;
    u = __ldg(slots + l * 1024);
  }
}

// The same for small bases, one thread per input in the order of Z.
template <bool INT>
__global__ void __launch_bounds__(256) k_ph_list(DevTables T, const double *WCC, int hL, int hR,
                                                 const int *exps, int gL, int gR, int kshift, double *Z) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const PhTerm p = t < T.n_ph ? T.ph_terms[t] : PhTerm{};
  const unsigned m = 0x0FFFFFFFu;
  pdl_go();
  pdl_wait();
  if (t >= T.n_ph) return;
  int k = 0;
  if (INT) {
    const int g = p.y >> 28 | (p.z >> 28) << 4 | (p.w >> 28) << 8;
    k = (exps[gL + g] - 1022) + (exps[gR + g] - 1022) - kshift;
  }
  Z[t] = ph_combine<INT>(WCC[p.x & m], WCC[p.y & m], WCC[p.z & m], WCC[p.w & m], (p.x >> 28) & 1, hL, hR, k);
}

// E0 = commutator_110 + commutator_220 (commutators.f90:10-33, 399-432) by one
// CTA of NT threads; the 220 sum arrives as the two-body kernel's per-CTA
// partials (e0p == nullptr: no 220 term).  Fixed order: strided per-thread
// sums, warp shuffles, then thread 0 adds the warp totals in index order.
// The partials were written by other CTAs, so they are read past L1.
constexpr int ENERGY_THREADS = 256;

template <int NT>
__device__ void energy_block(const DevTables &T, const double *L, int hL, const double *R, int hR, double *RES,
                             const double *e0p, int ne0p) {
  __shared__ double sh[2][NT / 32];
  const int A = T.A, P = T.P, tid = threadIdx.x;
  const double *Lph = L + T.off_fph, *Rph = R + T.off_fph;
  double v0 = 0.0, v1[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k = tid; k < P * A; k += NT) {
    int ji = T.orb[T.hole_orb[k / P]].x;
    v0 += (Lph[k] * Rph[k] * hL - Rph[k] * Lph[k] * hR) * (ji + 1);
  }
  if (e0p) {  // four independent chains, so the partials' loads overlap
    int k = tid;
    for (; k + 3 * NT < ne0p; k += 4 * NT) {
#pragma unroll
      for (int u = 0; u < 4; u++) v1[u] += __ldcg(e0p + k + u * NT);
    }
    for (; k < ne0p; k += NT) v1[0] += __ldcg(e0p + k);
  }
  v0 = warp_sum(v0);
  const double s1 = warp_sum((v1[0] + v1[1]) + (v1[2] + v1[3]));
  if ((tid & 31) == 0) {
    sh[0][tid >> 5] = v0;
    sh[1][tid >> 5] = s1;
  }
  __syncthreads();
  if (tid == 0) {
    double a = 0.0, c = 0.0;
    for (int w = 0; w < NT / 32; w++) {
      a += sh[0][w];
      c += sh[1][w];
    }
    RES[0] = a + c * 2.0;
  }
}

// Every two-body element of RES once (upper triangles of square arrays, the
// mirror written alongside): the one-body insertions of commutator_122, the
// antisymmetrised ladder epilogue of 222_pp_hh (:658-764) and the 222_ph
// recoupling sum over J' of {6j} Z(J').  Thread t takes element w0 + t of the
// work order `heads` while below w1.  PRE: the 122 part is already in RES
// (sums_122), and the split engine's nexps block exponents are cleared for the
// next commutator (nothing reads them any more).  The first n1 CTAs finish the
// one-body elements instead (one_body_221).  has220 (the allocation-free path, w0 = 0): each CTA leaves
// its commutator_220 partial in e0p for k_energy.
template <bool PRE>
__global__ void __launch_bounds__(ASM2_THREADS) k_assemble_2body(DevTables T, const double *__restrict__ L, int hL,
                                                                 const double *__restrict__ R, int hR,
                                                                 const double *W1, const double *W2, const double *Z,
                                                                 double *RES, int hRES,
                                                                 const Asm2Head *__restrict__ heads, long w0, long w1,
                                                                 int has220, double *e0p, int *exps, int nexps,
                                                                 int n1) {
  __shared__ double sh220[ASM2_THREADS / 32];
  if ((int)blockIdx.x < n1) {
    pdl_go();
    pdl_wait();
    one_body_221(T, hL, hR, W1, W2, RES, hRES, blockIdx.x);
    return;
  }
  const int cta = (int)blockIdx.x - n1;
  const long w = w0 + (long)cta * blockDim.x + threadIdx.x;
  const Asm2Head h = w < w1 ? heads[w] : Asm2Head{};
  pdl_go();
  pdl_wait();
  if (PRE && cta == 0)
    for (int i = threadIdx.x; i < nexps; i += ASM2_THREADS) exps[i] = 0;
  double e220 = 0.0;  // this element's commutator_220 term (pphh arrays only)
  if (w < w1) {
    const unsigned long long *tm = T.asm2_terms + h.start;
    const unsigned meta = h.meta;
    const int nL = hL < 0, nR = hR < 0, nres = hRES < 0, npm = (hL * hR) < 0;
    const int nd = (meta >> 18) & 3;
    const bool diag = (meta >> 20) & 1, square = (meta >> 21) & 1;
    const long e = h.e, em = h.em;
    double t;
    if (PRE) {
      t = RES[e];
    } else {
      t = sum122<1, 1>(tm, meta & 31, L, nL, R, nR);
      // / sqrt(1 + delta_ab) / sqrt(1 + delta_cd)
      if (nd) t = t * (nd == 1 ? 0.7071067811865476 : 0.5);
      if (diag) t = dflip(t, nres);
    }
    t = t + W1[e];
    t = t - W2[e];
    if (square) t = t - dflip(W1[em] - W2[em], npm);
    if ((meta >> 15) & 1) {
      const int n_in = (meta >> 5) & 31, n_out = (meta >> 10) & 31;
      const double *z = Z + h.zs, *s1 = T.six + h.six1, *s2 = T.six + h.six2;
      const double *zo = (meta >> 23) & 1 ? z : z + n_in;
      double a1 = 0.0, a2 = 0.0;
      for (int k = 0; k < n_in; k++) a1 = fma(s1[k], z[k], a1);
      for (int k = 0; k < n_out; k++) a2 = fma(s2[k], zo[k], a2);
      double sm = dflip(a1, (meta >> 16) & 1) + dflip(a2, (meta >> 24) & 1);
      // the reference's truncated 1/sqrt(2) literal for identical orbits
      if (nd) sm = sm * (nd == 1 ? .70710678118 : .70710678118 * .70710678118);
      t = t + sm;
    }
    if (diag) {
      RES[e] = dflip(t, nres);
    } else {
      RES[e] = t;
      if (square) RES[em] = dflip(t, nres);
    }
    // commutator_220 (commutators.f90:409-427): -(2J+1) L_pphh R_pphh herm_R
    if (has220 && ((meta >> 22) & 1)) e220 = -L[e] * R[e] * hR * (h.J2 + 1.0);
  }
  if (has220) {  // per-CTA partial in a fixed order
    e220 = warp_sum(e220);
    if ((threadIdx.x & 31) == 0) sh220[threadIdx.x >> 5] = e220;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t220 = 0.0;
      for (int k = 0; k < (int)(blockDim.x >> 5); k++) t220 += sh220[k];
      e0p[cta] = t220;
    }
  }
}

// E0 for the allocation-free path: one CTA over the two-body kernel's partials.
__global__ void __launch_bounds__(ENERGY_THREADS) k_energy(DevTables T, const double *L, int hL, const double *R,
                                                           int hR, double *RES, const double *e0p, int ne0p) {
  energy_block<ENERGY_THREADS>(T, L, hL, R, hR, RES, e0p, ne0p);
}

// E0 = commutator_110 + commutator_220 (commutators.f90:10-33, 399-432)
// straight from L and R: the 220 sum needs only their pphh arrays, so E0 runs
// beside the assembly kernels instead of after them.  One CTA; warp w takes
// the (2J,Tz,pi) blocks w, w + 16, ... in turn; fixed summation order.
constexpr int E0_THREADS = 512;

__global__ void __launch_bounds__(E0_THREADS) k_e0(DevTables T, const double *__restrict__ L, int hL,
                                                   const double *__restrict__ R, int hR, double *RES, int has220) {
  __shared__ double sh[2][E0_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int A = T.A, P = T.P;
  const double *Lph = L + T.off_fph, *Rph = R + T.off_fph;
  double v0 = 0.0, c = 0.0;
  for (int k = tid; k < P * A; k += E0_THREADS) {
    const int ji = T.orb[T.hole_orb[k / P]].x;
    v0 += (Lph[k] * Rph[k] * hL - Rph[k] * Lph[k] * hR) * (ji + 1);
  }
  if (has220)
    for (int q = wid; q < T.nblocks; q += E0_THREADS / 32) {
      const int n = T.gam_n1[q * 6 + 2] * T.gam_n2[q * 6 + 2];
      const double *Lq = L + T.gam_off[q * 6 + 2], *Rq = R + T.gam_off[q * 6 + 2];
      double s = 0.0;
      for (int k = lane; k < n; k += 32) s = fma(Lq[k], Rq[k], s);
      c += (T.blk_J2[q] + 1.0) * warp_sum(s);
    }
  v0 = warp_sum(v0);
  if (lane == 0) {
    sh[0][wid] = v0;
    sh[1][wid] = c;
  }
  __syncthreads();
  if (tid == 0) {
    double a = 0.0, cc = 0.0;
    for (int w = 0; w < E0_THREADS / 32; w++) {
      a += sh[0][w];
      cc += sh[1][w];
    }
    // 2 sum_q (2J+1) sum -L_pphh R_pphh herm_R
    RES[0] = a - 2.0 * hR * cc;
  }
}

// The one-body assembly in one launch, after the products.  ALL: in one pass, else
// in the two of the shared launches (front.cuh), so that every path of one basis
// and precision gives the same bits.
template <bool ALL>
__global__ void __launch_bounds__(FRONT_THREADS, ALL ? 10 : 8) k_one_body(DevTables T, SumsArgs a, const double *__restrict__ W1,
                                                            const double *__restrict__ W2) {
  one_body_front<ALL>(T, a, blockIdx.x, W1, W2);
  if (!ALL && (int)blockIdx.x < T.n_asm1_heavy) one_body_221(T, a.hL, a.hR, W1, W2, a.RES, a.hRES, blockIdx.x);
}

}  // namespace

int launch_front(imsrg_basis *b, const double *L, int hL, const double *R, int hR, const Front &f, cudaStream_t st) {
  FrontArgs a{};
  int *exps = nullptr, gL = 0, gR = 0, ncc = 0;
  if (f.p1 > f.p0) IMSRG_TRY(ozaki_chunks(b, f.p0, f.p1, &a.chunks, &a.nexp, &a.exps));
  if (f.sides) {
    ncc = (int)((b->cc_total + CC_THREADS - 1) / CC_THREADS);
    if (f.split) IMSRG_TRY(ozaki_cc_exponents(b, &exps, &gL, &gR));
  }
  const int grid = a.nexp + ncc;
  if (grid == 0) return IMSRG_OK;
  ProfScope ps(b, f.sides ? IMSRG_KERNEL_CC_FORWARD : IMSRG_KERNEL_OZAKI_SLICE, st);
  auto *kernel = f.sides == 0 ? k_front<0> : f.sides == 1 ? k_front<1> : f.sides == 2 ? k_front<2> : k_front<3>;
  kernel<<<grid, CC_THREADS, 0, st>>>(b->T, L, hL, R, hR, b->lcc, b->rcc, exps, gL, gR, a);
  b->launches++;
  return cuda_status(cudaGetLastError());
}

int launch_sums_122(imsrg_basis *b, const SumsArgs &a, cudaStream_t st) {
  const int grid = sums_122_ctas(b);
  if (grid == 0) return IMSRG_OK;
  ProfScope ps(b, IMSRG_KERNEL_ASSEMBLE_2BODY, st);
  k_sums_122<<<grid, FRONT_THREADS, 0, st>>>(b->T, a);
  b->launches++;
  return cuda_status(cudaGetLastError());
}

int launch_gemm_fp64(imsrg_basis *b, const double *L, int hL, const double *R, int hR) {
  if (b->ntiles == 0) return IMSRG_OK;
  Operands ops{};
  ops.src[SRC_L] = L;
  ops.src[SRC_R] = R;
  ops.src[SRC_W1] = b->w1;
  ops.src[SRC_W2] = b->w2;
  ops.src[SRC_LCC] = b->lcc;
  ops.src[SRC_RCC] = b->rcc;
  ops.src[SRC_WCC] = b->wcc;
  ops.dst[SRC_W1] = b->w1;
  ops.dst[SRC_W2] = b->w2;
  ops.dst[SRC_WCC] = b->wcc;
  ProfScope ps(b, IMSRG_KERNEL_GEMM_FP64);
  b->launches++;
  return cuda_status(launch_after(b->pdl, k_gemm_fp64<false>, b->ntiles, GT_THREADS, 0, b->stream, b->d_probs, b->d_tiles, ops,
                                  hL, hR, nullptr));
}

void gemm_fp64_plan(std::vector<GemmProb> &probs, int num_sms) {
  std::vector<GemmShape> sh;
  for (const GemmProb &p : probs) sh.push_back({p.M, p.N, (long)p.K * p.nterms, 0});
  gemm_split(sh, num_sms);
  for (size_t i = 0; i < probs.size(); i++) probs[i].split = sh[i].split;
}

std::vector<GemmTile> gemm_fp64_tiles(const std::vector<GemmProb> &probs) {
  std::vector<GemmShape> sh;
  for (const GemmProb &p : probs) sh.push_back({p.M, p.N, (long)p.K * p.nterms, p.split});
  return gemm_tiles(sh);
}

// Every problem keeps its own basis's K split, so a merged launch gives the
// bits of the single ones.
int gemm_fp64_merged(imsrg_basis *const *bases, int n, const double *const *L, const double *const *R,
                     GemmMerged *out) {
  std::vector<GemmProb> all;
  for (int i = 0; i < n; i++) {
    imsrg_basis *b = bases[i];
    const double *src[7] = {L[i], R[i], b->w1, b->w2, b->lcc, b->rcc, b->wcc};
    double *dst[7] = {nullptr, nullptr, b->w1, b->w2, nullptr, nullptr, b->wcc};
    for (GemmProb p : b->probs) {
      for (int t = 0; t < p.nterms; t++) {
        p.t[t].a_abs = src[p.t[t].a_src] + p.t[t].a_off;
        p.t[t].b_abs = src[p.t[t].b_src] + p.t[t].b_off;
      }
      p.c_abs = dst[p.c_dst] + p.c_off;
      p.inst = i;
      all.push_back(p);
    }
  }
  *out = GemmMerged();
  const std::vector<GemmTile> tiles = gemm_fp64_tiles(all);
  if (tiles.empty()) return IMSRG_OK;
  auto up = [](const void *h, size_t bytes, void **d) -> int {
    IMSRG_CUDA_TRY(cudaMalloc(d, bytes));
    return cuda_status(cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice));
  };
  int s = up(all.data(), all.size() * sizeof(GemmProb), (void **)&out->d_probs);
  if (s == IMSRG_OK) s = up(tiles.data(), tiles.size() * sizeof(GemmTile), (void **)&out->d_tiles);
  if (s != IMSRG_OK) {
    out->release();
    return s;
  }
  out->ntiles = (int)tiles.size();
  return IMSRG_OK;
}

int launch_gemm_fp64_merged(const GemmMerged &g, int hL, int hR, const int *act, cudaStream_t st) {
  if (g.ntiles == 0) return IMSRG_OK;
  Operands ops{};
  k_gemm_fp64<true><<<g.ntiles, GT_THREADS, 0, st>>>(g.d_probs, g.d_tiles, ops, hL, hR, act);
  return cuda_status(cudaGetLastError());
}

// exps == nullptr: WCC holds FP64 (the FP64 path and the split engine's FP64
// class), else the split engine's int64 level sums
static int ph_inputs(imsrg_basis *b, const double *WCC, int hL, int hR, const int *exps, int gL, int gR, int kshift,
                     double *Z, cudaStream_t st) {
  if (b->T.n_ph == 0) return IMSRG_OK;
  auto *kernel = b->T.ph_terms ? (exps ? k_ph_list<true> : k_ph_list<false>)
                               : (exps ? k_ph_patches<true> : k_ph_patches<false>);
  const unsigned grid = b->T.ph_terms ? (b->T.n_ph + 255) / 256 : 4 * b->T.n_ph_patches;
  b->launches++;
  return cuda_status(launch_after(b->pdl, kernel, grid, 256, 0, st, b->T, WCC, hL, hR, exps, gL, gR, kshift, Z));
}

int launch_ph_inputs(imsrg_basis *b, int hL, int hR, int precision) {
  const int *exps = nullptr;
  int gL = 0, gR = 0, kshift = 0;
  if (precision == IMSRG_PREC_OZAKI) IMSRG_TRY(ozaki_wcc_scale(b, &exps, &gL, &gR, &kshift));
  return ph_inputs(b, b->wcc, hL, hR, exps, gL, gR, kshift, b->zph, b->stream);
}

int launch_asm2_range(imsrg_basis *b, const double *L, int hL, const double *R, int hR, double *RES, int hRES,
                      long w0, long w1, bool by_range, int *exps, int nexps, bool one_body) {
  const int n1 = one_body ? b->T.n_asm1_heavy : 0;
  const long grid = n1 + (std::max(w1 - w0, 0L) + ASM2_THREADS - 1) / ASM2_THREADS;
  if (grid > 0) {
    IMSRG_CUDA_TRY(launch_after(b->pdl, k_assemble_2body<true>, (unsigned)grid,
                                ASM2_THREADS, 0, b->stream, b->T, L, hL, R, hR, b->w1, b->w2, b->zph, RES, hRES,
                                by_range ? b->T.asm2_head_out : b->T.asm2_head, w0, w1, 0, nullptr, exps, nexps,
                                n1));
    b->launches++;
  }
  return cuda_status(cudaGetLastError());
}

int launch_one_body(imsrg_basis *b, const SumsArgs &a, bool all, cudaStream_t st) {
  const int grid = one_body_ctas(b->T);
  if (grid == 0) return IMSRG_OK;
  ProfScope ps(b, IMSRG_KERNEL_ASSEMBLE_1BODY, st);
  (all ? k_one_body<true> : k_one_body<false>)<<<grid, FRONT_THREADS, 0, st>>>(b->T, a, b->w1, b->w2);
  b->launches++;
  return cuda_status(cudaGetLastError());
}

int launch_e0(imsrg_basis *b, const double *L, int hL, const double *R, int hR, double *RES, cudaStream_t st) {
  ProfScope ps(b, IMSRG_KERNEL_ASSEMBLE_1BODY, st);
  k_e0<<<1, E0_THREADS, 0, st>>>(b->T, L, hL, R, hR, RES, hL * hR == -1);
  b->launches++;
  return cuda_status(cudaGetLastError());
}

// The four FP64 launches of one commutator with caller-chosen workspace and
// stream; used by the allocation-free entry point (noalloc.cu).  Allocates
// nothing and records no profiling events.
int launch_commutator_fp64_ws(imsrg_basis *b, const Workspace &ws, const double *L, int hL, const double *R, int hR,
                              double *RES, int hRES, int with_e0, cudaStream_t st) {
  if (b->cc_total > 0) {
    k_front<3><<<(unsigned)((b->cc_total + CC_THREADS - 1) / CC_THREADS), CC_THREADS, 0, st>>>(
        b->T, L, hL, R, hR, ws.lcc, ws.rcc, nullptr, 0, 0, FrontArgs{});
    b->launches++;
  }
  if (b->ntiles > 0) {
    Operands ops{};
    ops.src[SRC_L] = L;
    ops.src[SRC_R] = R;
    ops.src[SRC_W1] = ws.w1;
    ops.src[SRC_W2] = ws.w2;
    ops.src[SRC_LCC] = ws.lcc;
    ops.src[SRC_RCC] = ws.rcc;
    ops.src[SRC_WCC] = ws.wcc;
    ops.dst[SRC_W1] = ws.w1;
    ops.dst[SRC_W2] = ws.w2;
    ops.dst[SRC_WCC] = ws.wcc;
    k_gemm_fp64<false><<<b->ntiles, GT_THREADS, 0, st>>>(b->d_probs, b->d_tiles, ops, hL, hR, nullptr);
    b->launches++;
  }
  IMSRG_TRY(ph_inputs(b, ws.wcc, hL, hR, nullptr, 0, 0, 0, ws.zph, st));
  const long n2 = b->T.n_asm2;
  if (n2 > 0) {
    const int has220 = with_e0 && hL * hR == -1;
    k_assemble_2body<false><<<asm2_ctas(b), ASM2_THREADS, 0, st>>>(b->T, L, hL, R, hR, ws.w1, ws.w2, ws.zph, RES, hRES,
                                                                  b->T.asm2_head, 0, n2, has220, ws.e0p, nullptr, 0, 0);
    b->launches++;
  }
  if (const int grid1 = one_body_ctas(b->T)) {
    k_one_body<true><<<grid1, FRONT_THREADS, 0, st>>>(b->T, SumsArgs{L, R, RES, hL, hR, hRES, 0}, ws.w1, ws.w2);
    b->launches++;
  }
  if (with_e0) {
    const bool e220 = hL * hR == -1;
    k_energy<<<1, ENERGY_THREADS, 0, st>>>(b->T, L, hL, R, hR, RES, e220 ? ws.e0p : nullptr, asm2_ctas(b));
    b->launches++;
  }
  return cuda_status(cudaGetLastError());
}

int preload_commutator_fp64_ws() {
  cudaFuncAttributes a;
  const void *fns[] = {(const void *)k_front<3>, (const void *)k_gemm_fp64<false>, (const void *)k_ph_list<false>,
                       (const void *)k_ph_patches<false>,
                       (const void *)k_assemble_2body<false>, (const void *)k_one_body<true>, (const void *)k_energy};
  for (const void *f : fns) {
    cudaError_t e = cudaFuncGetAttributes(&a, f);
    if (e != cudaSuccess) return cuda_status(e);
  }
  return IMSRG_OK;
}

}  // namespace imsrg
