// front.cuh -- the parts of a commutator that need only L and R, as CTA
// functions, so that a launch can hold several of them by CTA range.
//
// On small bases a split commutator is a chain of small kernels whose links set its
// time: about one microsecond where a kernel has one predecessor (and overlaps
// its end, launch_after), 2.4 where it waits for two.  There everything that may
// run together shares a launch, five in a row with E0 beside them:
//   exponents of L and R, Pandya transform | slicing, the sums below | products |
//   recoupling inputs | one-body assembly, two-body assembly
// (20.6 -> 18.5 us at emax 2, 31.3 -> 28.8 at emax 4; batch of twelve 438 -> 432).
// On large ones (more than kPhList two-body elements) and in FP64 the parts run as
// branches: the 122 sums then gate the products, and one-body work beside them or
// ahead of the assembly costs more than the links (side by side on one GPU: emax 5
// 42.8 us, merged 45.1; emax 6 104, merged 106-112; FP64 at emax 2 15.9, merged 16.4;
// from GPU to GPU the branches read 43 to 47, 104 to 109 and 16.0 to 17.8).
#pragma once

#include "device.cuh"

namespace imsrg {

constexpr int FRONT_THREADS = 128;

// commutator_111, 121 (one-body) and 122 (two-body) of RES: the last n1 CTAs the
// one-body elements, the others share the 122 sums.
struct SumsArgs {
  const double *L, *R;
  double *RES;
  int hL, hR, hRES, n1;
};

// commutator_122 (commutators.f90:283-396) of one element: f_L V_R - f_R V_L
// over its leg terms (term k at tm[k * STRIDE]), U terms in flight: their gathers
// and the next U terms are loaded before the first is used
template <int STRIDE, int U>
__device__ __forceinline__ double sum122(const unsigned long long *tm, int n122, const double *L, int nL,
                                         const double *R, int nR) {
  double t = 0.0;
  unsigned long long next[U];
#pragma unroll
  for (int i = 0; i < U; i++) next[i] = i < n122 ? tm[i * STRIDE] : 0;
  for (int k = 0; k < n122; k += U) {
    unsigned long long u[U];
    double vR[U], vL[U], fL[U], fR[U];
#pragma unroll
    for (int i = 0; i < U; i++) {
      u[i] = next[i];
      if (k + U + i < n122) next[i] = tm[(k + U + i) * STRIDE];
      if (i == 0 || k + i < n122) {
        const long vi = (long)(u[i] & 0xFFFFFFFull), fi = (long)((u[i] >> 28) & 0xFFFFFull);
        vR[i] = R[vi];
        vL[i] = L[vi];
        fL[i] = L[fi];
        fR[i] = R[fi];
      }
    }
#pragma unroll
    for (int i = 0; i < U; i++) {
      if (i > 0 && k + i >= n122) break;
      const int sg = (int)(u[i] >> 48) & 1, nsq = (int)(u[i] >> 49) & 3, tr = (int)(u[i] >> 51) & 1,
                ftr = (int)(u[i] >> 52) & 1;
      double a = dflip(vR[i], tr & nR), b = dflip(vL[i], tr & nL);
      if (nsq) {
        const double c = nsq == 1 ? IMSRG_SQRT2 : 2.0000000000000004;
        a = a * c;
        b = b * c;
      }
      t = fma(dflip(fL[i], (ftr & nL) ^ sg), a, t);
      t = fma(dflip(fR[i], (ftr & nR) ^ sg ^ 1), b, t);
    }
  }
  return t;
}

// The commutator_122 part of every two-body element (upper triangles), with
// the element's 1/sqrt(1 + delta) factors and the diagonal's sign, into RES:
// it needs only L and R, so it runs ahead of the products, and the assembly
// after them (k_assemble_2body<true>) starts from it.  One warp per 32
// elements of equal term count; term k of every lane is one coalesced load.
// The arithmetic is the assembly's own, so RES is bit-identical either way.
// (Packing the sqrt(2)-scaled (L, R) pairs first, for one 16-byte gather per
// term, measured slower here: the pack kernel took more of the shared front
// than it saved.)  What bounds it: the FP64 pipe (two FMAs a term) and its
// gathers.  It has time until the products are done, so half of the SMs' warp
// slots are enough and the kernels before the products find the other half free:
// with a CTA per four groups it took every slot first (emax = 6, five digits:
// 112.4 us per commutator, 109.5 with eight CTAs per SM, 111.5 with six or
// twelve; host call 203 -> 194, two flow steps 3440 -> 3250, FP64 493 -> 487).
// They gate the products all the same, whose CTAs each want a whole SM (four
// CTAs per SM 122 us, two 147), with loads as their longest stall: two terms in
// flight take 108.4 to 106.1 us, three or four 108.8 and 111.2.
constexpr int kPreCtas = 8;
__device__ __forceinline__ void sums_122(const DevTables &T, const SumsArgs &a, int cta, int ctas) {
  const int lane = threadIdx.x & 31;
  for (int g = (int)((cta * blockDim.x + threadIdx.x) >> 5); g < T.n_pre_warps; g += (int)(ctas * blockDim.x >> 5)) {
    const unsigned pe = T.pre_el[(long)g * 32 + lane];
    if (pe >> 31) continue;  // padding
    const Asm2PreWarp W = T.pre_warp[g];
    double t = sum122<32, 2>(T.pre_terms + W.base + lane, W.n122, a.L, a.hL < 0, a.R, a.hR < 0);
    const int nd = (pe >> 28) & 3;
    if (nd) t = t * (nd == 1 ? 0.7071067811865476 : 0.5);
    if ((pe >> 30) & 1) t = dflip(t, a.hRES < 0);
    a.RES[pe & 0x0FFFFFFFu] = t;
  }
}

// One-body element e: its array (0 fhh, 1 fph, 2 fpp), place and orbits.
struct OneBody {
  int type, p, q, pk, qk;
};
__device__ __forceinline__ OneBody one_body(const DevTables &T, long e) {
  const int A = T.A, P = T.P;
  const long nA2 = (long)A * A, nPA = (long)P * A;
  int type, p, q, pk, qk;
  if (e < nA2) {
    type = 0;
    p = (int)(e % A);
    q = (int)(e / A);
    pk = T.hole_orb[p];
    qk = T.hole_orb[q];
  } else if (e < nA2 + nPA) {
    type = 1;
    p = (int)((e - nA2) % P);
    q = (int)((e - nA2) / P);
    pk = T.part_orb[p];
    qk = T.hole_orb[q];
  } else {
    type = 2;
    p = (int)((e - nA2 - nPA) % P);
    q = (int)((e - nA2 - nPA) / P);
    pk = T.part_orb[p];
    qk = T.part_orb[q];
  }
  return {type, p, q, pk, qk};
}
__device__ __forceinline__ long one_body_at(const DevTables &T, const OneBody &o) {
  return (o.type == 0 ? T.off_fhh : o.type == 1 ? T.off_fph : T.off_fpp) + o.p + (long)o.q * (o.type == 0 ? T.A : T.P);
}

__device__ __forceinline__ void one_body_mirror(const DevTables &T, const OneBody &o, double *RES, int hRES, double x) {
  if (o.type == 1 || o.p == o.q) return;
  RES[one_body_at(T, o) + (o.q - o.p) + (long)(o.p - o.q) * (o.type == 0 ? T.A : T.P)] = x * hRES;
}

// One term of a commutator_221 sum; the second kind enters with -herm_L herm_R.
__device__ __forceinline__ double term_221(const OneBodyTerm &t, int npm, const double *W1, const double *W2) {
  const double w = ((t.meta & 8) ? W2 : W1)[t.idx] * t.coef;
  return (t.meta & 3) == 3 ? dflip(w, npm) : w;
}

// One-body assembly.  The (l,j,tz)-allowed upper-triangle elements carry the
// 121 and 221 gather lists (a few hundred independent terms each) and get a
// CTA of four warps; every other element only has the four commutator_111 dot
// products and gets one warp, four elements per CTA.  Each thread folds its
// partial dot products and gather sums into the element's final linear
// combination, so one reduction per element remains:
//   type 0: v0 + v1 hL - (v2 hL + v3) hR      type 1: v0 + v1 - v2 - v3
//   type 2: v0 hR + v1 - (v2 + v3 hR) hL
// plus (v4 + v5) / (2j_p + 1) on allowed elements, v4 the 121 sum, v5 the 221
// one.  The 221 sum alone needs the products: the shared launches form the rest, two
// thirds of the terms and all the dot products, ahead of them and add the 221 sum
// with one_body_221 (as one kernel after the products it was the last to end).
// Elsewhere it is added here (ALL, after the products), with one reduction less.
template <bool ALL>
__device__ __forceinline__ void one_body_front(const DevTables &T, const SumsArgs &a, int cta, const double *W1,
                                               const double *W2) {
  __shared__ double sh[4];
  const int A = T.A, P = T.P, hL = a.hL, hR = a.hR;
  const double *L = a.L, *R = a.R;
  const double *Lhh = L + T.off_fhh, *Lph = L + T.off_fph, *Lpp = L + T.off_fpp;
  const double *Rhh = R + T.off_fhh, *Rph = R + T.off_fph, *Rpp = R + T.off_fpp;
  const bool whole = cta < T.n_asm1_heavy;  // CTA-uniform
  long e;
  int tid, nt;
  if (whole) {
    e = T.asm1_heavy[cta];
    tid = threadIdx.x;
    nt = blockDim.x;
  } else {
    const int li = (cta - T.n_asm1_heavy) * 4 + (int)(threadIdx.x >> 5);
    if (li >= T.n_asm1_light) return;
    e = T.asm1_light[li];
    tid = threadIdx.x & 31;
    nt = 32;
  }
  const OneBody o = one_body(T, e);
  const int type = o.type, p = o.p, q = o.q;
  // commutator_111 (commutators.f90:36-80): four dot products
  double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (type == 0) {  // th1 = Lhh Rhh, th2 = Lph^T Rph
    for (int k = tid; k < A; k += nt) {
      v[0] = fma(Lhh[p + (long)k * A], Rhh[k + (long)q * A], v[0]);
      v[2] = fma(Lhh[q + (long)k * A], Rhh[k + (long)p * A], v[2]);
    }
    for (int k = tid; k < P; k += nt) {
      v[1] = fma(Lph[k + (long)p * P], Rph[k + (long)q * P], v[1]);
      v[3] = fma(Lph[k + (long)q * P], Rph[k + (long)p * P], v[3]);
    }
  } else if (type == 1) {  // Lph Rhh + Lpp Rph - Rph Lhh - Rpp Lph
    for (int k = tid; k < A; k += nt) {
      v[0] = fma(Lph[p + (long)k * P], Rhh[k + (long)q * A], v[0]);
      v[2] = fma(Rph[p + (long)k * P], Lhh[k + (long)q * A], v[2]);
    }
    for (int k = tid; k < P; k += nt) {
      v[1] = fma(Lpp[p + (long)k * P], Rph[k + (long)q * P], v[1]);
      v[3] = fma(Rpp[p + (long)k * P], Lph[k + (long)q * P], v[3]);
    }
  } else {  // tp1 = Lph Rph^T, tp2 = Lpp Rpp
    for (int k = tid; k < A; k += nt) {
      v[0] = fma(Lph[p + (long)k * P], Rph[q + (long)k * P], v[0]);
      v[2] = fma(Lph[q + (long)k * P], Rph[p + (long)k * P], v[2]);
    }
    for (int k = tid; k < P; k += nt) {
      v[1] = fma(Lpp[p + (long)k * P], Rpp[k + (long)q * P], v[1]);
      v[3] = fma(Lpp[q + (long)k * P], Rpp[k + (long)p * P], v[3]);
    }
  }
  double v5 = 0.0;
  if (whole) {  // the gather list: commutator_121, and 221 behind it
    const int st = T.obt_start[e], n = ALL ? T.obt_count[e] : T.obt_121[e];
    const int nL = hL < 0, nR = hR < 0, npm = hL * hR > 0;
    for (int k = tid; k < n; k += nt) {
      const OneBodyTerm t = T.obt[st + k];
      const int kind = t.meta & 3;
      if (ALL && kind >= 2) {
        v5 += term_221(t, npm, W1, W2);
        continue;
      }
      const int tr = (t.meta >> 2) & 1, ph = t.meta >> 8;
      const double rv = dflip(R[t.idx], tr & nR) * t.coef;
      const double lv = dflip(L[t.idx], tr & nL) * t.coef;
      const double lph = Lph[ph], rph = Rph[ph];
      if (kind == 0) {  // L_ai (herm_L R) - R_ai (herm_R L) at <a p|i q>
        v[4] = fma(dflip(lph, nL), rv, v[4]);
        v[4] = fma(-dflip(rph, nR), lv, v[4]);
      } else {  // -L_ai R + R_ai L at <i p|a q>
        v[4] = fma(-lph, rv, v[4]);
        v[4] = fma(rph, lv, v[4]);
      }
    }
  }
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
  double x = fma(c3, v[3], fma(c2, v[2], fma(c1, v[1], c0 * v[0])));
  const double rj = 1.0 / (T.orb[o.pk].x + 1.0);
  if (whole) x = fma(rj, v[4], x);
  if (ALL && whole) x = fma((type != 1 && p == q) ? a.hRES * rj : rj, v5, x);
  x = warp_sum(x);
  if (whole) {
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    x = ((sh[0] + sh[1]) + sh[2]) + sh[3];
  }
  if (tid != 0) return;
  a.RES[one_body_at(T, o)] = x;
  if (ALL && whole) one_body_mirror(T, o, a.RES, a.hRES, x);
}

__device__ __forceinline__ void sums_cta(const DevTables &T, const SumsArgs &a, int cta, int ctas) {
  const int n = ctas - a.n1;
  if (cta < n) sums_122(T, a, cta, n);
  else one_body_front<false>(T, a, cta - n, nullptr, nullptr);
}
// CTAs of each (of FRONT_THREADS threads)
inline int one_body_ctas(const DevTables &T) { return T.n_asm1_heavy + (T.n_asm1_light + 3) / 4; }
inline int sums_122_ctas(const imsrg_basis *b) {
  return (int)std::min(((long)b->T.n_pre_warps * 32 + FRONT_THREADS - 1) / FRONT_THREADS, (long)kPreCtas * b->num_sms);
}

// Adds commutator_221 to allowed element number cta (see one_body_front), where a
// diagonal of fhh or fpp takes it times herm(RES) (((t + s121) hRES + s221) hRES
// with hRES^2 = 1), and mirrors it.
__device__ __forceinline__ void one_body_221(const DevTables &T, int hL, int hR, const double *W1, const double *W2,
                                             double *RES, int hRES, int cta) {
  __shared__ double sh[4];
  const long e = T.asm1_heavy[cta];
  const OneBody o = one_body(T, e);
  const long at = one_body_at(T, o);
  const double x0 = threadIdx.x == 0 ? RES[at] : 0.0;
  const int st = T.obt_start[e], n = T.obt_count[e], npm = hL * hR > 0;
  double v = 0.0;
  for (int k = T.obt_121[e] + (int)threadIdx.x; k < n; k += blockDim.x) v += term_221(T.obt[st + k], npm, W1, W2);
  const double rj = 1.0 / (T.orb[o.pk].x + 1.0);
  v = warp_sum(v * ((o.type != 1 && o.p == o.q) ? hRES * rj : rj));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x != 0) return;
  const double x = x0 + (((sh[0] + sh[1]) + sh[2]) + sh[3]);
  RES[at] = x;
  one_body_mirror(T, o, RES, hRES, x);
}

}  // namespace imsrg
