// adjoint.cu -- reverse-mode derivatives: the adjoint of the commutator and of
// the Magnus flow.
//
// The commutator RES = [X, Y] (the sequence of IMSRG_MAGNUS.f90:207-219,
// commutators.f90:10-925) is bilinear.  For a fixed X its adjoint with
// respect to Y is the transposed linear map
//     Ybar = d<Cbar, [X, Y]> / dY,
// built here by transposing every piece of the forward kernels
// (kernels_comm.cu) on the same host-built gather lists, one kernel per
// piece, in the reverse order of the forward data flow:
//   1. k_adj_prep, everything that needs only X and Cbar: the ladder epilogue
//      of 222_pp_hh hands Cbar to W1bar / W2bar and to the commutator_122
//      sums' weights, the 222_ph recoupling to Zbar, LCC is X's Pandya transform;
//   2. k_adj_122: the commutator_122 insertions to Ybar (two- and one-body, on
//      transposed gather lists) and the recoupling inputs^T, Zbar to WCCbar;
//   3. k_adj_one: one-body assembly^T (commutator_111 / 121 to Ybar, 221 to
//      W1bar / W2bar) and the energy's 110 and 220 terms;
//   4. every dense product transposed as one grouped FP64 launch: the twelve
//      ladder products of each block into Ybar's two-body arrays, and
//      RCCbar = WCCbar^T LCC per cross-coupled block;
//   5. Pandya transform^T (calculate_cross_coupled, cross_coupled.f90:
//      1190-1300): RCCbar back to Ybar.
// The adjoint with respect to X follows from antisymmetry, [X, Y] = -[Y, X]:
//     d<Cbar, [X, Y]> / dX = -(the adjoint above with the roles swapped).
// The one-body and Pandya lists become scatters, added with FP64
// atomics: the adjoint's results agree run to run to rounding, not bit for bit
// (the forward commutator stays atomic-free and bit-reproducible).
//
// The flow's adjoint (imsrg_gpu_magnus_decouple_adjoint) records one Magnus
// flow (the host-driven sequence of magnus_decouple, IMSRG_MAGNUS.f90:15-128,
// with MAGNUS_EXPAND :622-693, euler_step :756-766, BCH_EXPAND :149-234 and
// build_gs_white, generators.f90:4-106) with every series term kept in device
// memory, then sweeps back from E0(s) through each step: BCH terms, the Euler
// step, the Magnus terms and the White generator.  One backward sweep gives
// the gradient of E0(s) with respect to every element of the input
// Hamiltonian, so dE0/dc_k for H(c) = T + sum_k c_k V_k is one dot product
// per parameter.  The reference has no derivative code; its checks are
// central finite differences of the flow.
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "front.cuh"
#include "gemm_fp64.cuh"

namespace imsrg {

namespace {

// ---------------------------------------------------------------------------
// Grouped FP64 products of the adjoint: C += sum_t alpha_t op(A_t) op(B_t),
// each term with its own contraction length (the transposed ladder products
// of one output array read different intermediates), in the forward's tiles
// (gemm_fp64.cuh).
// ---------------------------------------------------------------------------
struct AdjTerm {
  int a_src, b_src, ta, tb;
  long a_off, b_off;
  int lda, ldb, K;
  double coef;
  int use_hl, use_hr;
};

constexpr int kAdjTerms = 6;
struct AdjProb {
  int M, N, nterms, c_dst;
  long c_off;
  int ldc;
  AdjTerm t[kAdjTerms];
};

// operands: X (the fixed operator), W1bar, W2bar, WCCbar, LCC; outputs: Ybar, RCCbar
enum { AS_X = 0, AS_W1 = 1, AS_W2 = 2, AS_WCC = 3, AS_LCC = 4, AD_Y = 0, AD_RCC = 1 };
struct AdjOps {
  const double *src[5];
  double *dst[2];
};

__global__ void __launch_bounds__(GT_THREADS, GT_CTAS) k_gemm_adj(const AdjProb *__restrict__ probs,
                                                         const GemmTile *__restrict__ tiles, AdjOps ops, int hL,
                                                         int hR) {
  const GemmTile t = tiles[blockIdx.x];
  const AdjProb &P = probs[t.prob];
  pdl_wait();
  gemm_cta_tile<true>(
      t,
      [&](int it, auto add) {
        const AdjTerm &m = P.t[it];
        add(ops.src[m.a_src] + m.a_off, m.ta ? (long)m.lda : 1L, m.ta ? 1L : (long)m.lda, ops.src[m.b_src] + m.b_off,
            m.tb ? (long)m.ldb : 1L, m.tb ? 1L : (long)m.ldb, m.K,
            (m.coef < 0) ^ (m.use_hl && hL < 0) ^ (m.use_hr && hR < 0));  // coefficients are +-1
      },
      P.nterms, P.M, P.N, ops.dst[P.c_dst] + P.c_off, P.ldc);
}

// ---------------------------------------------------------------------------
// 1 and 2. Two-body assembly^T (k_assemble_2body's sequence read backwards).
// Forward, per element e with mirror em:
//      t0 = s122 * nd;  t1 = diag ? -t0 (herm(RES) < 0) : t0;
//      t2 = t1 + W1[e] - W2[e] - [square] (+-)(W1[em] - W2[em]) + sm;
//      RES[e] = diag ? +-t2 : t2;  RES[em] = herm(RES) t2 (square, off-diagonal)
// The commutator_122 sums s122 = sum fL vR + fR vL are transposed on lists of
// their own, one per two-body element of Y and one per one-body element, so
// nothing scatters: as scatters, five million atomics fell on a few hundred
// one-body elements (324 us at emax = 6, 39 us at emax = 4; k_adj_122 takes 55
// and 15 us with the recoupling inputs^T in it, which took 23 and 5).  Work
// that depends on the same inputs shares a launch, by CTA range: five launches
// instead of seven and six memsets (emax = 4: 119 -> 63 us, emax = 6: 850 -> 567).
// The particle-hole part (Zbar, LCC, WCCbar, then RCCbar's product) and the rest
// (weights, 122 sums, one-body assembly^T, then the ladder products) meet only in
// the Pandya transform^T, so they run on two streams, each with its share of the
// first two kernels' CTA ranges: 63.5 -> 53.5 us at emax = 4, where the chain of
// launches is the time, and 560 -> 548 at emax = 6, where both halves want the
// FP64 pipe (a high-priority second stream 557, three product CTAs per SM beside
// it 552).  On each stream a kernel is launched as the dependent of the one before
// it, which saves a link's launch latency (53.0 -> 48.4 us, 548 -> 544), but starts
// as that one ends: started earlier (pdl_go), its CTAs held slots the other stream
// wanted (51.4 us).
// ---------------------------------------------------------------------------

// Gather lists of the transposed sums (host-built from the forward's).
struct AdjLists {
  const int *mir;             // per two-body flat index from off_2b: partner (bits 0-27), 28 upper or diagonal, 29
                              // diagonal, 30 square array
  const int4 *quad;           // per orbit quadruple: first head, heads, first Z, inside Zs
  const Asm2Head *qhead;      // heads in quadruple order
  const int *zquad;           // quadruple of each Z
  const Asm2PreWarp *v_warp;  // two-body targets: 32 to a warp, n entries each (as DevTables::pre_warp)
  const int *v_el;            // target, -1 pads
  const unsigned long long *v_terms;  // bits 0-27 element e, 28-47 one-body f, 48 sign, 51 V transposed, 52 f transposed
  int n_v_warps;
  const unsigned long long *f_terms;  // one-body targets: bits 0-27 element e, 28-55 V, 56 sign, 57-58 sqrt(2)
                                      // factors, 59 V transposed, 60 f transposed
  const int2 *f_chunk;        // first entry and entries of each chunk
  int n_f_chunks;
  const int4 *f_target;       // one-body flat index, first chunk, chunks
  int n_f_targets;
};
constexpr int ADJ_THREADS = 256, ADJ_F_CHUNK = 2048, ADJ_ZERO = 2048;

// d(t2) of the element whose stored index is e (upper or diagonal) from Cbar
__device__ __forceinline__ double adj_tb(const double *__restrict__ Cb, long e, long em, bool square, int nres) {
  if (!square) return Cb[e];
  return e == em ? dflip(Cb[e], nres) : Cb[e] + dflip(Cb[em], nres);
}

// CTAs (from `first` on) [0, n0): W1bar, W2bar = -W1bar and the 122 weights U, by
// flat index, and zeros to Ybar's E0 and one-body part; [n0, n1): Zbar; [n1, n2):
// LCC; the rest zero RCCbar.
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_prep(DevTables T, AdjLists A, const double *__restrict__ X,
                                                          int hL, int hR, const double *__restrict__ Cb, int hRES,
                                                          long off_2b, int first, int n0, int n1, int n2,
                                                          double *W1b, double *W2b, double *U, double *Zb,
                                                          double *LCC, double *RCCb, double *Yb) {
  const int nres = hRES < 0;
  const int blk = blockIdx.x + first;
  if (blk < n0) {
    const long i = (long)blk * ADJ_THREADS + threadIdx.x;
    if (i >= T.nfull) return;
    if (i < off_2b) {
      Yb[i] = 0.0;
      return;
    }
    const int m = A.mir[i - off_2b];
    const long p = m & 0x0FFFFFFF;
    const bool upper = (m >> 28) & 1, diag = (m >> 29) & 1, square = (m >> 30) & 1;
    const int npm = (hL * hR) < 0;
    const double tb = upper ? adj_tb(Cb, i, p, square, nres) : adj_tb(Cb, p, i, square, nres);
    double w = tb;
    if (diag) w = tb - dflip(tb, npm);
    else if (!upper) w = -dflip(tb, npm);
    W1b[i] = w;
    W2b[i] = -w;
    double u = diag ? dflip(tb, nres) : tb;
    const int nd = T.vsq[i];  // identical orbit pairs
    if (nd) u = u * (nd == 1 ? 0.7071067811865476 : 0.5);
    U[i] = u;
    return;
  }
  if (blk < n1) {
    const long t = (long)(blk - n0) * ADJ_THREADS + threadIdx.x;
    if (t >= T.n_ph) return;
    const int4 q = A.quad[A.zquad[t]];
    const int k = (int)t - q.z;
    double z = 0.0;
    for (int h = q.x; h < q.x + q.y; h++) {
      const Asm2Head H = A.qhead[h];
      const int nd = (H.meta >> 18) & 3;
      double s = adj_tb(Cb, H.e, H.em, (H.meta >> 21) & 1, nres);
      if (nd) s = s * (nd == 1 ? .70710678118 : .70710678118 * .70710678118);
      const bool shared = (H.meta >> 23) & 1;  // the outside channel reads the inside Z
      if (k < q.w) z = fma(dflip(s, (H.meta >> 16) & 1), T.six[H.six1 + k], z);
      if (shared || k >= q.w) z = fma(dflip(s, (H.meta >> 24) & 1), T.six[H.six2 + (shared ? k : k - q.w)], z);
    }
    Zb[t] = z;
    return;
  }
  if (blk < n2) {
    const long t = (long)(blk - n1) * ADJ_THREADS + threadIdx.x;
    if (t >= T.cc_total) return;
    const int v = T.ccf_order[t];
    const long e = T.ccf_packed ? (v & 0xFFFFFF) : v;
    double s = 0.0;
    for (int k = T.cct_start[e]; k < T.cct_start[e + 1]; k++) {
      const int ix = T.cct_idx[k];
      s = fma(T.cct_coef[k], dflip(X[ix & 0x7fffffff], ((unsigned)ix >> 31) & (hL < 0)), s);
    }
    LCC[e] = s;
    return;
  }
  const long z0 = (long)(blk - n2) * ADJ_ZERO;
  for (long i = z0 + threadIdx.x; i < min(z0 + ADJ_ZERO, (long)T.cc_total); i += ADJ_THREADS) RCCb[i] = 0.0;
}

// Recoupling inputs^T, a quarter of a patch of a block's (x, y) plane
// (k_ph_patches): every entry of WCCbar belongs to one (x, y) of the patches, as
// W(x,y), W(y',x'), W(x',y') or W(y,x), or as several of them at once, so the
// patches write the whole plane, zeros included, without atomics.
__device__ __forceinline__ void adj_ph(const DevTables &T, const double *Zb, int hL, int hR, double *WCCb,
                                       int quarter) {
  const PhPatch &p = T.ph_patch[quarter >> 2];
  const int lane = threadIdx.x & 31, ty = (threadIdx.x >> 5) + (quarter & 3) * 8, rl = p.rlen;
  const int x = p.x0 + lane, y = p.y0 + ty;
  // only the form that the patches hold
  if (x >= p.half || y >= rl || (y >= p.half ? y - p.half : y) < x) return;
  double *W = WCCb + p.w, *V = WCCb + p.v;
  const bool one = p.w == p.v;
  const unsigned char *ph = T.cc_rowph + p.row0;
  const int nph = __ldg(ph + x) ^ __ldg(ph + y), xr = ph_rev(p, x), yr = ph_rev(p, y);
  double z = 0.0;
  for (int l = 0; l < p.layers; l++) {
    const unsigned u = __ldg(T.ph_slots + ((long)p.table + l) * 1024 + ty * 32 + lane);
    if ((u & kPhSlot) != kPhNone) z += dflip(Zb[u & kPhSlot], ((u & kPhFlip) != 0) ^ ((u & kPhSwap) && hL * hR > 0));
  }
  const double c1 = dflip(z, hL < 0), c4 = -dflip(z, hR < 0);  // W(x, y), W(y, x)
  const double c2 = dflip(c1, nph), c3 = dflip(c4, nph);       // W(y', x'), W(x', y')
  double v1 = c1, v2 = c2, v3 = c3, v4 = c4;
  if (x == y) {
    v1 += c4;
    v4 = v1;
    v2 += c3;
    v3 = v2;
  }
  if (one && x == yr) {
    const double t1 = v1 + v2, t3 = v3 + v4;
    v1 = v2 = t1;
    v3 = v4 = t3;
  }
  if (one && x == xr && y == yr && x != y) {
    const double t1 = v1 + v3, t2 = v2 + v4;
    v1 = v3 = t1;
    v2 = v4 = t2;
  }
  W[x + (long)y * rl] = v1;
  V[xr + (long)yr * rl] = v3;
  V[yr + (long)xr * rl] = v2;
  W[y + (long)x * rl] = v4;
}

// CTAs (from `first` on) [0, n0): the partial sum of one chunk of a one-body
// target's list; [n0, n1): two-body targets, a warp per 32 (sets Ybar there); the rest: the
// recoupling inputs^T.
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_122(DevTables T, AdjLists A, const double *__restrict__ X, int hL,
                                                         int hR, const double *U, const double *Zb, int first,
                                                         int n0, int n1, double *fpart, double *WCCb, double *Yb) {
  __shared__ double sh[32];
  pdl_wait();
  const int nL = hL < 0, nR = hR < 0;
  const int blk = blockIdx.x + first;
  if (blk < n0) {
    const int2 c = A.f_chunk[blk];
    double s = 0.0;
    for (int k = threadIdx.x; k < c.y; k += ADJ_THREADS) {
      const unsigned long long u = A.f_terms[(long)c.x + k];
      const long e = (long)(u & 0xFFFFFFFull), vi = (long)((u >> 28) & 0xFFFFFFFull);
      const int sg = (int)(u >> 56) & 1, nsq = (int)(u >> 57) & 3, tr = (int)(u >> 59) & 1, ftr = (int)(u >> 60) & 1;
      double v = X[vi];
      if (nsq) v = v * (nsq == 1 ? IMSRG_SQRT2 : 2.0000000000000004);
      s = fma(dflip(U[e], (tr & nL) ^ (ftr & nR) ^ sg ^ 1), v, s);
    }
    s = block_sum_ops(s, sh);
    if (threadIdx.x == 0) fpart[blk] = s;
    return;
  }
  if (blk < n1) {
    const int g = (blk - n0) * (ADJ_THREADS / 32) + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (g >= A.n_v_warps) return;
    const int vi = A.v_el[(long)g * 32 + lane];
    if (vi < 0) return;  // padding
    const Asm2PreWarp W = A.v_warp[g];
    const unsigned long long *tm = A.v_terms + W.base + lane;
    double s = 0.0;
    for (int k = 0; k < W.n122; k++) {
      const unsigned long long u = tm[k * 32];
      if (u >> 63) break;  // the lane's list has ended
      const long e = (long)(u & 0xFFFFFFFull), fi = (long)((u >> 28) & 0xFFFFFull);
      const int sg = (int)(u >> 48) & 1, tr = (int)(u >> 51) & 1, ftr = (int)(u >> 52) & 1;
      s = fma(dflip(U[e], (tr & nR) ^ (ftr & nL) ^ sg), X[fi], s);
    }
    const int nsq = T.vsq[vi];
    if (nsq) s = s * (nsq == 1 ? IMSRG_SQRT2 : 2.0000000000000004);
    Yb[vi] = s;
    return;
  }
  adj_ph(T, Zb, hL, hR, WCCb, blk - n1);
}

// ---------------------------------------------------------------------------
// 3. One-body assembly^T over the one-body assembly's work split (an allowed
//    upper-triangle element per CTA, every other element per warp).  Forward:
//      x = c0 v0 + c1 v1 + c2 v2 + c3 v3 + [allowed] (rj v4 + c5 v5)
//    with v0..v3 the commutator_111 dot products, v4 the 121 sums, v5 the 221
//    sums; RES[p, q] = x and, for allowed square elements, RES[q, p] = herm x.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void adj_1body(const DevTables &T, const double *X, int hL, int hR,
                                          const double *__restrict__ Cb, int hRES, double *Yb, double *W1b,
                                          double *W2b) {
  const int A = T.A, P = T.P;
  const double *Lhh = X + T.off_fhh, *Lph = X + T.off_fph, *Lpp = X + T.off_fpp;
  double *Rhh = Yb + T.off_fhh, *Rph = Yb + T.off_fph, *Rpp = Yb + T.off_fpp;
  const int nheavy = T.n_asm1_heavy;
  const bool whole = (int)blockIdx.x < nheavy;
  long e;
  int tid, nt;
  if (whole) {
    e = T.asm1_heavy[blockIdx.x];
    tid = threadIdx.x;
    nt = blockDim.x;
  } else {
    const int li = ((int)blockIdx.x - nheavy) * 4 + (int)(threadIdx.x >> 5);
    if (li >= T.n_asm1_light) return;
    e = T.asm1_light[li];
    tid = threadIdx.x & 31;
    nt = 32;
  }
  const OneBody o = one_body(T, e);
  const int type = o.type, p = o.p, q = o.q;
  // whole: the (l, j, tz)-allowed elements of the upper triangles
  const long at = one_body_at(T, o);
  double xb = Cb[at];
  if (whole && type != 1 && p != q) xb += hRES * Cb[at + (q - p) + (long)(p - q) * (type == 0 ? A : P)];
  if (xb == 0.0) return;
  double c0 = 1.0, c1 = 1.0, c2 = -1.0, c3 = -1.0;
  if (type == 0) {
    c1 = hL;
    c2 = -(double)(hL * hR);
    c3 = -hR;
  } else if (type == 2) {
    c0 = hR;
    c2 = -hL;
    c3 = -(double)(hR * hL);
  }
  const double b0 = c0 * xb, b1 = c1 * xb, b2 = c2 * xb, b3 = c3 * xb;
  // commutator_111 (commutators.f90:36-80), the Y factor of each product
  if (type == 0) {
    for (int k = tid; k < A; k += nt) {
      atomicAdd(Rhh + k + (long)q * A, b0 * Lhh[p + (long)k * A]);
      atomicAdd(Rhh + k + (long)p * A, b2 * Lhh[q + (long)k * A]);
    }
    for (int k = tid; k < P; k += nt) {
      atomicAdd(Rph + k + (long)q * P, b1 * Lph[k + (long)p * P]);
      atomicAdd(Rph + k + (long)p * P, b3 * Lph[k + (long)q * P]);
    }
  } else if (type == 1) {
    for (int k = tid; k < A; k += nt) {
      atomicAdd(Rhh + k + (long)q * A, b0 * Lph[p + (long)k * P]);
      atomicAdd(Rph + p + (long)k * P, b2 * Lhh[k + (long)q * A]);
    }
    for (int k = tid; k < P; k += nt) {
      atomicAdd(Rph + k + (long)q * P, b1 * Lpp[p + (long)k * P]);
      atomicAdd(Rpp + p + (long)k * P, b3 * Lph[k + (long)q * P]);
    }
  } else {
    for (int k = tid; k < A; k += nt) {
      atomicAdd(Rph + q + (long)k * P, b0 * Lph[p + (long)k * P]);
      atomicAdd(Rph + p + (long)k * P, b2 * Lph[q + (long)k * P]);
    }
    for (int k = tid; k < P; k += nt) {
      atomicAdd(Rpp + k + (long)q * P, b1 * Lpp[p + (long)k * P]);
      atomicAdd(Rpp + k + (long)p * P, b3 * Lpp[q + (long)k * P]);
    }
  }
  if (!whole) return;
  // commutator_121 (:83-280) and 221 (:435-578) terms
  const double rj = 1.0 / (T.orb[o.pk].x + 1.0);
  const double u4 = rj * xb, u5 = ((type != 1 && p == q) ? hRES * rj : rj) * xb;
  const int st = T.obt_start[e], n = T.obt_count[e];
  const int nL = hL < 0, nR = hR < 0, npm = hL * hR > 0;
  for (int k = tid; k < n; k += nt) {
    const OneBodyTerm t = T.obt[st + k];
    const int kind = t.meta & 3;
    if (kind < 2) {
      const int tr = (t.meta >> 2) & 1, ph = t.meta >> 8;
      const double lv = dflip(X[t.idx], tr & nL) * t.coef;
      const double lph = Lph[ph];
      if (kind == 0) {  // L_ai (herm_L R) - R_ai (herm_R L) at <a p|i q>
        atomicAdd(Yb + t.idx, dflip(u4 * dflip(lph, nL) * t.coef, tr & nR));
        atomicAdd(Rph + ph, -dflip(u4 * lv, nR));
      } else {  // -L_ai R + R_ai L at <i p|a q>
        atomicAdd(Yb + t.idx, -dflip(u4 * lph * t.coef, tr & nR));
        atomicAdd(Rph + ph, u4 * lv);
      }
    } else {
      double *Wb = (t.meta & 8) ? W2b : W1b;
      const double w = u5 * t.coef;
      atomicAdd(Wb + t.idx, kind == 3 ? dflip(w, npm) : w);
    }
  }
}

// CTAs [0, n0): the one-body assembly^T; [n0, n1): the one-body targets of the
// commutator_122 lists, their chunks in order; [n1, n2): commutator_110^T, E0 +=
// sum_ai (2j_i+1) (L_ai R_ai herm_L - R_ai L_ai herm_R); the rest, a CTA per (2J,
// Tz, pi) block: commutator_220^T, E0 -= 2 herm_R (2J+1) L_pphh R_pphh.
__global__ void __launch_bounds__(128) k_adj_one(DevTables T, AdjLists A, const double *X, int hL, int hR,
                                                 const double *__restrict__ Cb, int hRES,
                                                 const double *fpart, int n0, int n1, int n2, double *Yb,
                                                 double *W1b, double *W2b) {
  pdl_wait();
  const int blk = blockIdx.x;
  if (blk < n0) {
    adj_1body(T, X, hL, hR, Cb, hRES, Yb, W1b, W2b);
  } else if (blk < n1) {
    const int t = (blk - n0) * 128 + threadIdx.x;
    if (t >= A.n_f_targets) return;
    const int4 f = A.f_target[t];
    double s = 0.0;
    for (int k = f.y; k < f.y + f.z; k++) s += fpart[k];
    atomicAdd(Yb + f.x, s);
  } else if (blk < n2) {
    const int k = (blk - n1) * 128 + threadIdx.x;
    if (k >= T.P * T.A) return;
    const int ji = T.orb[T.hole_orb[k / T.P]].x;
    atomicAdd(Yb + T.off_fph + k, Cb[0] * (double)(hL - hR) * (ji + 1) * X[T.off_fph + k]);
  } else {
    const int q = blk - n2, n = T.gam_n1[q * 6 + 2] * T.gam_n2[q * 6 + 2];
    const long o = T.gam_off[q * 6 + 2];
    for (int k = threadIdx.x; k < n; k += 128)
      atomicAdd(Yb + o + k, -2.0 * hR * (T.blk_J2[q] + 1.0) * Cb[0] * X[o + k]);
  }
}

// 5. Pandya transform^T: RCC[e] = sum_k coef_k (herm_R if transposed) R[idx_k]
__global__ void __launch_bounds__(256) k_adj_cc(DevTables T, const double *__restrict__ RCCb, int hR, double *Yb) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= T.cc_total) return;
  const double r = RCCb[e];
  if (r == 0.0) return;
  const int nR = hR < 0;
  for (int k = T.cct_start[e]; k < T.cct_start[e + 1]; k++) {
    const int ix = T.cct_idx[k];
    const int tr = (int)((unsigned)ix >> 31), idx = ix & 0x7fffffff;
    atomicAdd(Yb + idx, T.cct_coef[k] * dflip(r, tr & nR));
  }
}

// Fixed-order dot product: per-CTA partials, then one CTA sums them in order.
constexpr int DOT_CTAS = 256, DOT_THREADS = 256;
__global__ void __launch_bounds__(DOT_THREADS) k_dot_partial(const double *__restrict__ x,
                                                             const double *__restrict__ y, long n, double *part) {
  __shared__ double sh[DOT_THREADS / 32];
  double s = 0.0;
  for (long i = (long)blockIdx.x * DOT_THREADS + threadIdx.x; i < n; i += (long)DOT_CTAS * DOT_THREADS)
    s = fma(x[i], y[i], s);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < DOT_THREADS / 32; k++) t += sh[k];
    part[blockIdx.x] = t;
  }
}

__global__ void k_dot_final(const double *__restrict__ part, double *out) {
  double t = 0.0;
  for (int k = 0; k < DOT_CTAS; k++) t += part[k];
  *out = t;
}

}  // namespace

// Per-basis state of the adjoint (built on first use; imsrg_basis::adjoint is set
// once all of it stands).
struct AdjState {
  double *w1b = nullptr, *w2b = nullptr, *rccb = nullptr, *wccb = nullptr, *zb = nullptr, *u = nullptr;
  double *fpart = nullptr;
  AdjLists lists{};
  AdjProb *d_probs = nullptr;
  GemmTile *d_tiles = nullptr;
  int ntiles = 0, nladder = 0;  // tiles: the ladder products', then RCCbar's
  cudaStream_t side = nullptr;  // the part without the particle-hole product
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};

namespace {

AdjState *adj_of(imsrg_basis *b) { return (AdjState *)b->adjoint; }

int adj_alloc(imsrg_basis *b, long n, double **out) {
  void *p = nullptr;
  IMSRG_CUDA_TRY(cudaMalloc(&p, (size_t)std::max(n, 1L) * sizeof(double)));
  b->dev_allocs.push_back(p);
  *out = (double *)p;
  return IMSRG_OK;
}

AdjTerm aterm(int a, long aoff, int lda, int ta, int bsrc, long boff, int ldb, int tb, int K, double coef,
              int hl = 0, int hr = 0) {
  AdjTerm t{};
  t.a_src = a;
  t.a_off = aoff;
  t.lda = lda;
  t.ta = ta;
  t.b_src = bsrc;
  t.b_off = boff;
  t.ldb = ldb;
  t.tb = tb;
  t.K = K;
  t.coef = coef;
  t.use_hl = hl;
  t.use_hr = hr;
  return t;
}

// The transposes of the forward products (basis.cpp's problem list, with
// R the variable): for each forward term alpha op(A) op(R) the adjoint adds
// alpha op(A)^T Wbar into Rbar, for alpha op(R) op(B) it adds alpha Wbar
// op(B)^T; the terms that land on one array of one block are one problem.
std::vector<AdjProb> adjoint_problems(const imsrg_basis *b) {
  std::vector<AdjProb> out;
  auto add = [&](int M, int N, int dst, long off, int ldc, std::initializer_list<AdjTerm> ts) {
    if (M <= 0 || N <= 0) return;
    AdjProb p{};
    p.M = M;
    p.N = N;
    p.c_dst = dst;
    p.c_off = off;
    p.ldc = ldc;
    for (const AdjTerm &t : ts)
      if (t.K > 0) p.t[p.nterms++] = t;
    if (p.nterms) out.push_back(p);
  };
  for (int qb = 0; qb < b->nblocks; qb++) {
    const int np = b->npp[qb], nb = b->nph[qb], nh = b->nhh[qb];
    auto G = [&](int g) { return b->gam_off[qb * 6 + g - 1]; };
    // pppp: W1_pppp = L1 R1, W1_pphh = -R1 L3, W1_ppph = -R1 L2
    add(np, np, AD_Y, G(1), np,
        {aterm(AS_X, G(1), np, 1, AS_W1, G(1), np, 0, np, 1.0), aterm(AS_W1, G(3), np, 0, AS_X, G(3), np, 1, nh, -1.0),
         aterm(AS_W1, G(2), np, 0, AS_X, G(2), np, 1, nb, -1.0)});
    // hhhh: W2_hhhh = L5 R5, W2_pphh = L3 R5, W2_phhh = L6 R5
    add(nh, nh, AD_Y, G(5), nh,
        {aterm(AS_X, G(5), nh, 1, AS_W2, G(5), nh, 0, nh, 1.0), aterm(AS_X, G(3), np, 1, AS_W2, G(3), np, 0, np, 1.0),
         aterm(AS_X, G(6), nb, 1, AS_W2, G(6), nb, 0, nb, 1.0)});
    // pphh: W1_hhhh = hL L3^T R3, W2_pppp = hR L3 R3^T, W1_pphh = L1 R3,
    // W2_pphh = -R3 L5, W1_phhh = hL L2^T R3, W2_ppph = -hL R3 L6^T
    add(np, nh, AD_Y, G(3), np,
        {aterm(AS_X, G(3), np, 0, AS_W1, G(5), nh, 0, nh, 1.0, 1, 0),
         aterm(AS_W2, G(1), np, 1, AS_X, G(3), np, 0, np, 1.0, 0, 1),
         aterm(AS_X, G(1), np, 1, AS_W1, G(3), np, 0, np, 1.0),
         aterm(AS_W2, G(3), np, 0, AS_X, G(5), nh, 1, nh, -1.0),
         aterm(AS_X, G(2), np, 0, AS_W1, G(6), nb, 0, nb, 1.0, 1, 0),
         aterm(AS_W2, G(2), np, 0, AS_X, G(6), nb, 0, nb, -1.0, 1, 0)});
    // ppph: W1_phph = hL L2^T R2, W1_ppph = L1 R2, W1_phhh = -hR R2^T L3
    add(np, nb, AD_Y, G(2), np,
        {aterm(AS_X, G(2), np, 0, AS_W1, G(4), nb, 0, nb, 1.0, 1, 0),
         aterm(AS_X, G(1), np, 1, AS_W1, G(2), np, 0, np, 1.0),
         aterm(AS_X, G(3), np, 0, AS_W1, G(6), nb, 1, nh, -1.0, 0, 1)});
    // phhh: W2_phph = hR L6 R6^T, W2_phhh = -R6 L5, W2_ppph = hR L3 R6^T
    add(nb, nh, AD_Y, G(6), nb,
        {aterm(AS_W2, G(4), nb, 1, AS_X, G(6), nb, 0, nb, 1.0, 0, 1),
         aterm(AS_W2, G(6), nb, 0, AS_X, G(5), nh, 1, nh, -1.0),
         aterm(AS_W2, G(2), np, 1, AS_X, G(3), np, 0, np, 1.0, 0, 1)});
  }
  // WCC = LCC RCC^T per cross-coupled block: RCCbar = WCCbar^T LCC
  for (int q1 = 0; q1 < b->ccblocks; q1++) {
    const int r = b->cc_rlen[q1], nb = b->cc_nph[q1];
    add(r, nb, AD_RCC, b->cc_off[q1], r, {aterm(AS_WCC, b->wcc_off[q1], r, 1, AS_LCC, b->cc_off[q1], r, 0, r, 1.0)});
  }
  return out;
}

}  // namespace

namespace {

template <typename V>
int adj_upload(imsrg_basis *b, const std::vector<V> &h, const V **out) {
  void *p = nullptr;
  IMSRG_CUDA_TRY(cudaMalloc(&p, std::max<size_t>(h.size() * sizeof(V), 16)));
  b->dev_allocs.push_back(p);
  if (!h.empty()) IMSRG_CUDA_TRY(cudaMemcpy(p, h.data(), h.size() * sizeof(V), cudaMemcpyHostToDevice));
  *out = (const V *)p;
  return IMSRG_OK;
}

// The transposed lists, from the forward's heads and commutator_122 terms.
int adj_lists(imsrg_basis *b, AdjState *a) {
  const DevTables &T = b->T;
  AdjLists &A = a->lists;
  std::vector<Asm2Head> heads(T.n_asm2);
  if (T.n_asm2)
    IMSRG_CUDA_TRY(cudaMemcpy(heads.data(), T.asm2_head, heads.size() * sizeof(Asm2Head), cudaMemcpyDeviceToHost));
  // by flat index: the entries of one target then run along matrix columns
  std::sort(heads.begin(), heads.end(), [](const Asm2Head &x, const Asm2Head &y) { return x.e < y.e; });
  long nt = 0;
  for (const Asm2Head &h : heads) nt = std::max(nt, (long)h.start + (long)(h.meta & 31));
  std::vector<unsigned long long> terms(nt);
  if (nt) IMSRG_CUDA_TRY(cudaMemcpy(terms.data(), T.asm2_terms, nt * 8, cudaMemcpyDeviceToHost));
  const long off = b->off_2b, n2 = b->nfull - off;
  // partner of every element
  std::vector<int> mir(n2, 0);
  for (const Asm2Head &h : heads) {
    const bool diag = (h.meta >> 20) & 1, square = (h.meta >> 21) & 1;
    mir[h.e - off] = (square ? h.em : h.e) | 1 << 28 | (diag ? 1 << 29 : 0) | (square ? 1 << 30 : 0);
    if (square && !diag) mir[h.em - off] = h.e | 1 << 30;
  }
  // heads by quadruple (the elements that share recoupling inputs)
  std::vector<Asm2Head> qhead;
  for (const Asm2Head &h : heads)
    if (((h.meta >> 15) & 1) && ((h.meta >> 5) & 1023)) qhead.push_back(h);
  std::stable_sort(qhead.begin(), qhead.end(), [](const Asm2Head &x, const Asm2Head &y) { return x.zs < y.zs; });
  std::vector<int4> quad;
  std::vector<int> zquad(T.n_ph, 0);
  for (size_t h = 0; h < qhead.size(); h++) {
    const int n_in = (qhead[h].meta >> 5) & 31, n_out = (qhead[h].meta >> 23) & 1 ? 0 : (qhead[h].meta >> 10) & 31;
    if (h == 0 || qhead[h].zs != qhead[h - 1].zs) {
      quad.push_back(make_int4((int)h, 0, qhead[h].zs, n_in));
      for (int k = 0; k < n_in + n_out; k++) zquad[qhead[h].zs + k] = (int)quad.size() - 1;
    }
    quad.back().y++;
  }
  // commutator_122 terms by two-body element of Y (grouped by count, 32 to a
  // warp) and by one-body element (chunks)
  std::vector<int> vn(n2, 0), fn(off, 0);
  for (const Asm2Head &h : heads)
    for (int k = 0; k < (int)(h.meta & 31); k++) {
      const unsigned long long u = terms[h.start + k];
      vn[(long)(u & 0xFFFFFFFull) - off]++;
      fn[(u >> 28) & 0xFFFFFull]++;
    }
  std::vector<int> order(n2);
  for (long i = 0; i < n2; i++) order[i] = (int)i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return vn[x] > vn[y]; });
  std::vector<Asm2PreWarp> vw;
  std::vector<int> ve;
  std::vector<long> vpos(n2);  // next entry of each target
  long nv = 0;
  for (long g = 0; g < n2; g += 32) {
    const int n = vn[order[g]];  // the warp's longest list; shorter ones end early
    vw.push_back({nv, n, 0});
    for (long l = 0; l < 32; l++) {
      ve.push_back(g + l < n2 ? (int)(order[g + l] + off) : -1);
      if (g + l < n2) vpos[order[g + l]] = nv + l;
    }
    nv += 32L * n;
  }
  std::vector<unsigned long long> vt(nv, ~0ull);  // padding: bit 63
  std::vector<long> fpos(off);
  std::vector<int2> chunk;
  std::vector<int4> target;
  long nf = 0;
  for (long f = 0; f < off; f++) {
    fpos[f] = nf;
    if (!fn[f]) continue;
    target.push_back(make_int4((int)f, (int)chunk.size(), 0, 0));
    for (int k = 0; k < fn[f]; k += ADJ_F_CHUNK) {
      chunk.push_back(make_int2((int)(nf + k), std::min(ADJ_F_CHUNK, fn[f] - k)));
      target.back().z++;
    }
    nf += fn[f];
  }
  if (nf >= (1L << 31)) return IMSRG_ERR_TOO_LARGE;
  std::vector<unsigned long long> ft(nf);
  for (const Asm2Head &h : heads)
    for (int k = 0; k < (int)(h.meta & 31); k++) {
      const unsigned long long u = terms[h.start + k];
      const unsigned long long v = u & 0xFFFFFFFull, f = (u >> 28) & 0xFFFFFull, e = (unsigned long long)h.e;
      vt[vpos[(long)v - off]] = (u & ~0xFFFFFFFull) | e;
      vpos[(long)v - off] += 32;
      ft[fpos[f]++] = e | v << 28 | ((u >> 48) & 1) << 56 | ((u >> 49) & 3) << 57 | ((u >> 51) & 1) << 59 |
                      ((u >> 52) & 1) << 60;
    }
  A.n_v_warps = (int)vw.size();
  A.n_f_chunks = (int)chunk.size();
  A.n_f_targets = (int)target.size();
  IMSRG_TRY(adj_upload(b, mir, &A.mir));
  IMSRG_TRY(adj_upload(b, quad, &A.quad));
  IMSRG_TRY(adj_upload(b, qhead, &A.qhead));
  IMSRG_TRY(adj_upload(b, zquad, &A.zquad));
  IMSRG_TRY(adj_upload(b, vw, &A.v_warp));
  IMSRG_TRY(adj_upload(b, ve, &A.v_el));
  IMSRG_TRY(adj_upload(b, vt, &A.v_terms));
  IMSRG_TRY(adj_upload(b, ft, &A.f_terms));
  IMSRG_TRY(adj_upload(b, chunk, &A.f_chunk));
  IMSRG_TRY(adj_upload(b, target, &A.f_target));
  return IMSRG_OK;
}

}  // namespace

namespace {

int adj_build(imsrg_basis *b, AdjState *a) {
  IMSRG_TRY(adj_alloc(b, b->nfull, &a->w1b));
  IMSRG_TRY(adj_alloc(b, b->nfull, &a->w2b));
  IMSRG_TRY(adj_alloc(b, b->cc_total, &a->rccb));
  IMSRG_TRY(adj_alloc(b, b->wcc_total, &a->wccb));
  IMSRG_TRY(adj_alloc(b, b->T.n_ph, &a->zb));
  IMSRG_TRY(adj_lists(b, a));
  IMSRG_TRY(adj_alloc(b, b->nfull, &a->u));
  IMSRG_TRY(adj_alloc(b, a->lists.n_f_chunks, &a->fpart));
  std::vector<AdjProb> probs = adjoint_problems(b);
  std::vector<GemmShape> shapes;
  for (const AdjProb &p : probs) {
    long k = 0;
    for (int t = 0; t < p.nterms; t++) k += p.t[t].K;
    shapes.push_back({p.M, p.N, k, 0});
  }
  gemm_split(shapes, b->num_sms);
  std::vector<GemmTile> tiles = gemm_tiles(shapes);
  a->ntiles = (int)tiles.size();
  a->nladder = (int)(std::stable_partition(tiles.begin(), tiles.end(), [&](const GemmTile &t) {
                       return probs[t.prob].c_dst == AD_Y;
                     }) - tiles.begin());
  IMSRG_CUDA_TRY(cudaStreamCreateWithFlags(&a->side, cudaStreamNonBlocking));
  IMSRG_CUDA_TRY(cudaEventCreateWithFlags(&a->ev_fork, cudaEventDisableTiming));
  IMSRG_CUDA_TRY(cudaEventCreateWithFlags(&a->ev_join, cudaEventDisableTiming));
  auto up = [&](const void *h, size_t bytes, void **d) -> int {
    IMSRG_CUDA_TRY(cudaMalloc(d, std::max<size_t>(bytes, 16)));
    b->dev_allocs.push_back(*d);
    return cuda_status(cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice));
  };
  IMSRG_TRY(up(probs.data(), probs.size() * sizeof(AdjProb), (void **)&a->d_probs));
  IMSRG_TRY(up(tiles.data(), tiles.size() * sizeof(GemmTile), (void **)&a->d_tiles));
  return IMSRG_OK;
}

void adj_delete(AdjState *a) {
  if (a->ev_fork) cudaEventDestroy(a->ev_fork);
  if (a->ev_join) cudaEventDestroy(a->ev_join);
  if (a->side) cudaStreamDestroy(a->side);
  delete a;  // device buffers are in b->dev_allocs
}

}  // namespace

// All or nothing: what a failed attempt allocated is given back, so that the next
// call fails or succeeds by itself.
int adjoint_prepare(imsrg_basis *b) {
  if (b->adjoint) return IMSRG_OK;
  AdjState *a = new (std::nothrow) AdjState();
  if (!a) return IMSRG_ERR_OOM;
  const size_t mark = b->dev_allocs.size();
  int s = IMSRG_ERR_OOM;
  try {
    s = adj_build(b, a);
  } catch (const std::bad_alloc &) {  // the host's lists
  }
  if (s != IMSRG_OK) {
    for (; b->dev_allocs.size() > mark; b->dev_allocs.pop_back()) cudaFree(b->dev_allocs.back());
    adj_delete(a);
    return s;
  }
  b->adjoint = a;
  return IMSRG_OK;
}

void adjoint_free(imsrg_basis *b) {
  if (b->adjoint) adj_delete(adj_of(b));
  b->adjoint = nullptr;
}

// Yb = d<Cb, [X, Y]> / dY for herm(X) = hX, herm(Y) = hY; with_e0 = 0: the
// commutator leaves RES E0 alone (as MAGNUS_EXPAND's do), so Cb[0] is ignored.
int commutator_adjoint_dev(imsrg_basis *b, const double *X, int hX, const double *Cb, int hY, int with_e0,
                           double *Yb) {
  IMSRG_TRY(adjoint_prepare(b));
  AdjState *a = adj_of(b);
  cudaStream_t st = b->stream;
  const int hL = hX, hR = hY, hRES = -hX * hY;
  const DevTables &T = b->T;
  const AdjLists &A = a->lists;
  ProfScope ps(b, IMSRG_KERNEL_OPS, st);
  auto ctas = [](long n, long per) { return (int)((n + per - 1) / per); };
  const bool serial = b->prof.on;
  cudaStream_t side = serial ? st : a->side;
  if (!serial) {
    IMSRG_CUDA_TRY(cudaEventRecord(a->ev_fork, st));
    IMSRG_CUDA_TRY(cudaStreamWaitEvent(side, a->ev_fork, 0));
  }
  const int p0 = ctas(b->nfull, ADJ_THREADS), p1 = p0 + ctas(T.n_ph, ADJ_THREADS),
            p2 = p1 + ctas(b->cc_total, ADJ_THREADS), p3 = p2 + ctas(b->cc_total, ADJ_ZERO);
  const int v0 = A.n_f_chunks, v1 = v0 + ctas(A.n_v_warps, ADJ_THREADS / 32), v2 = v1 + 4 * T.n_ph_patches;
  cudaError_t err = cudaSuccess;
  auto prep = [&](int from, int to, cudaStream_t s) {
    if (to == from) return;
    k_adj_prep<<<to - from, ADJ_THREADS, 0, s>>>(T, A, X, hL, hR, Cb, hRES, b->off_2b, from, p0, p1, p2, a->w1b,
                                                 a->w2b, a->u, a->zb, b->lcc, a->rccb, Yb);
    b->launches++;
  };
  auto sums = [&](int from, int to, cudaStream_t s) {
    if (to == from) return;
    err = err ? err : launch_after(true, k_adj_122, to - from, ADJ_THREADS, 0, s, T, A, X, hL, hR, a->u, a->zb, from, v0,
                                   v1, a->fpart, a->wccb, Yb);
    b->launches++;
  };
  AdjOps ops{};
  ops.src[AS_X] = X;
  ops.src[AS_W1] = a->w1b;
  ops.src[AS_W2] = a->w2b;
  ops.src[AS_WCC] = a->wccb;
  ops.src[AS_LCC] = b->lcc;
  ops.dst[AD_Y] = Yb;
  ops.dst[AD_RCC] = a->rccb;
  auto products = [&](int from, int to, cudaStream_t s) {
    if (to == from) return;
    err = err ? err : launch_after(true, k_gemm_adj, to - from, GT_THREADS, 0, s, a->d_probs, a->d_tiles + from, ops, hL,
                                   hR);
    b->launches++;
  };
  // (while kernel timing is on, one stream; the order below holds there too)
  prep(0, p0, side);
  prep(p0, p3, st);
  sums(v1, v2, st);
  products(a->nladder, a->ntiles, st);
  sums(0, v1, side);
  {
    const int n0 = T.n_asm1_heavy + (T.n_asm1_light + 3) / 4, n1 = n0 + ctas(A.n_f_targets, 128),
              n2 = n1 + (with_e0 ? ctas((long)b->P * b->A, 128) : 0),
              n3 = n2 + (with_e0 && hL * hR == -1 ? b->nblocks : 0);
    if (n3) {
      err = err ? err : launch_after(true, k_adj_one, n3, 128, 0, side, T, A, X, hL, hR, Cb, hRES, a->fpart, n0, n1, n2,
                                     Yb, a->w1b, a->w2b);
      b->launches++;
    }
  }
  products(0, a->nladder, side);
  IMSRG_CUDA_TRY(err);
  if (!serial) {
    IMSRG_CUDA_TRY(cudaEventRecord(a->ev_join, side));
    IMSRG_CUDA_TRY(cudaStreamWaitEvent(st, a->ev_join, 0));
  }
  if (b->cc_total > 0) {
    k_adj_cc<<<(unsigned)((b->cc_total + 255) / 256), 256, 0, st>>>(b->T, a->rccb, hR, Yb);
    b->launches++;
  }
  return cuda_status(cudaGetLastError());
}

// <x, y> over n doubles in a fixed order, into host memory.
int dot_dev(imsrg_basis *b, const double *x, const double *y, long n, double *out) {
  if (!b->dot_part) IMSRG_TRY(adj_alloc(b, DOT_CTAS + 1, &b->dot_part));
  double *dot = b->dot_part + DOT_CTAS;
  k_dot_partial<<<DOT_CTAS, DOT_THREADS, 0, b->stream>>>(x, y, n, b->dot_part);
  k_dot_final<<<1, 1, 0, b->stream>>>(b->dot_part, dot);
  b->launches += 2;
  IMSRG_CUDA_TRY(cudaMemcpyAsync(b->h_scal, dot, sizeof(double), cudaMemcpyDeviceToHost, b->stream));
  IMSRG_CUDA_TRY(cudaStreamSynchronize(b->stream));
  *out = b->h_scal[0];
  return IMSRG_OK;
}

int adjoint_monob(imsrg_basis *b, double **out) {
  if (!b->monob) IMSRG_TRY(adj_alloc(b, (long)b->norb * b->norb, &b->monob));
  *out = b->monob;
  return IMSRG_OK;
}

}  // namespace imsrg
