// fx.cuh -- SU(3) products of FP64 data on the integer pipe.
//
// GB300 runs 2 FP64 multiply-adds per clock and SM (measured 1.7-2.0), but 59 `mad.wide.s32` (32 x 32 + 64
// bits), and the two pipes run side by side (measured: 8 mad.wide and one FP64 fma per iteration take the
// fma's time alone).  Links are bounded by one, so a matrix product can run in 60-bit fixed point with
// one exponent per matrix: three mad.wide per real multiply-add instead of one FP64 fma, about ten times the
// rate, and an error of ~2^-58 of the matrices' size against FP64's ~2^-54.
//
// A number is q 2^(e-60), q a 64-bit integer kept in two halves, q = h 2^32 + 2 l with -2^30 <= l < 2^30, and
// e the exponent of its matrix; |q| < 2^63, so a value may reach 8 2^e.  A product of two numbers is
//   h h' 2^64 + (h l' + l h') 2^33   (l l' 2^2 dropped: < 2^-58 of 2^(e+e'))
// summed in two 64-bit accumulators: six terms of |h h'| <= 2^58 and twelve of |h l'| <= 2^59 fit easily.
// Sums of q are exact modulo 2^64, so an intermediate sum may wrap where the final one is in range.
//
// Links near the identity keep their relative accuracy: a link is held as A = U - 1 with the exponent of
// its largest entry (link_near), and a product of links as w = ab - 1 = A + B + AB.  The plaquette's
// anti-Hermitian part is then accurate to ~2^-57 of the links' departure from 1, as small as that may be,
// where FP64's is to ~2^-53 of it.
//
// What the format cannot hold is found, not assumed away: a link entry above 1.03 (or not finite), a row of a
// product of two links whose norm is not near one, an accumulator or a sum of two or three out of range set Guard, and the
// caller runs the FP64 arithmetic for that site instead.
#pragma once

#include "su3.cuh"

namespace glasma {
namespace fx {

typedef long long ll;

struct R {
  int h, l;
};
struct C {
  R re, im;
};
struct M {
  C e[9];  // e[i + 3*j]
};
struct Acc {
  ll hh, cr;
};
// extremes of what has to stay in range, in one comparison at the end
struct Guard {
  int hi, lo;
  bool bad;
};

constexpr int kScale = 60;
constexpr int kOneH = 1 << (kScale - 32);  // h of the value 1 at exponent 0

__device__ __forceinline__ R split(ll q) {
  const int lo = (int)q, hi = (int)(q >> 32);
  R r;
  r.h = hi - (lo >> 31);
  r.l = lo >> 1;
  return r;
}
__device__ __forceinline__ ll join(const R& r) { return ((ll)r.h << 32) + 2 * (ll)r.l; }

__device__ __forceinline__ Acc acc_zero() {
  Acc a;
  a.hh = 0;
  a.cr = 0;
  return a;
}
// half a unit of the result, so that finish rounds
__device__ __forceinline__ Acc acc_half() {
  Acc a;
  a.hh = 0;
  a.cr = 1 << 26;
  return a;
}
__device__ __forceinline__ void mad(Acc& s, const R& a, const R& b) {
  s.hh += (ll)a.h * b.h;
  s.cr += (ll)a.h * b.l;
  s.cr += (ll)a.l * b.h;
}
__device__ __forceinline__ ll finish(const Acc& s) { return (s.hh << 4) + (s.cr >> 27); }
__device__ __forceinline__ ll finish_diff(const Acc& p, const Acc& n) {
  Acc s;
  s.hh = p.hh - n.hh;
  s.cr = p.cr - n.cr;
  return finish(s);
}
// The accumulated value stays below 4: |hh| < 2^58, its high word below 2^26.
__device__ __forceinline__ void watch(Guard& g, ll hh_re, ll hh_im) {
  const int a = (int)(hh_re >> 32), b = (int)(hh_im >> 32);
  g.hi = max(g.hi, max(a, b));
  g.lo = min(g.lo, min(a, b));
}
__device__ __forceinline__ bool tripped(const Guard& g) { return g.bad || g.hi >= (1 << 26) || g.lo < -(1 << 26); }
__device__ __forceinline__ Guard guard_init() {
  Guard g;
  g.hi = 0;
  g.lo = 0;
  g.bad = false;
  return g;
}

// ---- doubles in and out -------------------------------------------------------------------------------
// By integer operations on the bits: GB300's FP64 <-> 64-bit integer conversions run on the FP64 pipe, at the
// rate of an fma (measured: with them the force kernel kept that pipe 67 % busy, two thirds of it converting).
// shift(k): what the conversions take for a scale of 2^k
__device__ __forceinline__ int shift(int k) { return 1083 - k; }
// |v| 2^k, truncated; |v| 2^k < 2^62 (larger values give garbage, never a fault)
__device__ __forceinline__ ll shifted(unsigned long long m, int by) {
  ll q;
  asm("shr.u64 %0, %1, %2;" : "=l"(q) : "l"(m), "r"(by));  // clamps: zero beyond 63
  return q;
}
__device__ __forceinline__ ll magnitude(double v, int sh) {
  const int h = __double2hiint(v);
  const unsigned long long m =
      ((unsigned long long)((h & 0xfffff) | 0x100000) << 40) | ((unsigned long long)(unsigned)__double2loint(v) << 8);
  return shifted(m, sh - ((h >> 20) & 0x7ff));
}
// A float times 2^76, exactly: subnormal numbers become normal ones, and a zero, taken for the smallest of those, falls below
// 2^-203, under the last place of every k up to 199 (kMinExpOf<float>).  (A double's smallest exponents are out of reach of
// every k in use.)  One multiplication of the FP32 pipe, which these kernels leave idle.
constexpr int kLift = 76;
__device__ __forceinline__ int lifted(float v) { return __float_as_int(v * 0x1p76f); }
__device__ __forceinline__ ll magnitude(float v, int sh) {
  const int h = lifted(v);
  return shifted((unsigned long long)((h & 0x7fffff) | 0x800000) << 37, sh - (896 - kLift) - ((h >> 23) & 0xff));
}
__device__ __forceinline__ int sign_word(double v) { return __double2hiint(v) >> 31; }
__device__ __forceinline__ int sign_word(float v) { return __float_as_int(v) >> 31; }
template <typename T>
__device__ __forceinline__ ll to_fixed(T v, int sh) {
  const ll q = magnitude(v, sh), s = sign_word(v);
  return (q ^ s) - s;
}
template <typename T>
__device__ __forceinline__ R to_fixed_split(T v, int sh) {
  R r = split(magnitude(v, sh));
  const int sg = sign_word(v) | 1;
  r.h *= sg;
  r.l *= sg;
  return r;
}
// q 2^k, rounded to nearest (half up)
__device__ __forceinline__ double from_fixed(ll q, int k) {
  const ll s = q >> 63;
  const unsigned long long m = (unsigned long long)((q ^ s) - s);
  const int n = __clzll((ll)m);
  const unsigned long long t = m << (n & 63);
  const unsigned long long b = (t >> 11) + ((t >> 10) & 1) + ((unsigned long long)(unsigned)(1023 + 62 + k - n) << 52);
  return m == 0 ? 0.0 : __longlong_as_double((ll)b | (q & (1LL << 63)));
}
// The same by two FP64 additions (q in two pieces placed into the low bits of 2^84 and 2^52) where that pipe has room:
// 9 operations instead of 24.
__device__ __forceinline__ double from_fixed_fp64(ll q, int k) {
  const double hi = __hiloint2double(0x45300000, (int)(q >> 32) ^ (int)0x80000000);
  const double lo = __hiloint2double(0x43300000, (int)q);
  const double v = (hi - 19342822341709703277445120.0) + lo;  // 2^84 + 2^63 + 2^52
  return q == 0 ? 0.0 : __hiloint2double(__double2hiint(v) + (int)((unsigned)k << 20), __double2loint(v));
}
// Exponents from here on: smaller values are held at 2^(kMinExp - 60).
template <typename T>
constexpr int kMinExpOf = sizeof(T) == 8 ? -900 : -139;
constexpr int kMinExp = kMinExpOf<double>;
// High words of numbers below 2^kMinExp (kHalf: 2^(kMinExp/2)) that are not zero: they would keep fewer than their digits, so
// FP64 takes them.  (Numbers below 2^-1042, whose high word is zero, count as zeros; every float is held.)
template <bool kHalf = false>
__device__ __forceinline__ bool tiny(int top) {
  return (unsigned)(top - 1) < (unsigned)((1022 + (kHalf ? kMinExp / 2 : kMinExp)) << 20) - 1;
}
// |v| < 2^exponent_of(largest |high word| of v)
__device__ __forceinline__ int exponent_of(int habs) { return (habs >> 20) - 1022; }
constexpr int kMaxEntryHi = 0x3FF07AE1;  // 1.03

// the high word of |v| as a double
__device__ __forceinline__ int habs(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ int habs(float v) { return ((lifted(v) & 0x7fffffff) >> 3) + ((896 - kLift) << 20); }

// A plain matrix with entries up to one (a link), exponent 0; kDag: its dagger.
template <bool kDag = false, typename T, typename I>
__device__ __forceinline__ void link_plain(const cx<T>* __restrict__ U, I S, int mu, I s, M& m, Guard& g) {
  const cx<T>* p = U + ((I)(mu * 9) * S + s);
  int top = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const cx<T> v = p[(I)(kDag ? k / 3 + 3 * (k % 3) : k) * S];
    top = max(top, max(habs(v.re), habs(v.im)));
    m.e[k].re = to_fixed_split(v.re, shift(kScale));
    m.e[k].im = to_fixed_split(kDag ? -v.im : v.im, shift(kScale));
  }
  g.bad |= top > kMaxEntryHi;
}

// A = U - 1 (dag: U^dagger - 1) with the exponent of its largest entry (at most 0).
template <typename T, typename I>
__device__ __forceinline__ void link_near(const cx<T>* __restrict__ U, I S, int mu, I s, M& m, int& e, Guard& g,
                                          bool dag = false) {
  const cx<T>* p = U + ((I)(mu * 9) * S + s);
  cx<T> v[9];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      cx<T> x = p[(I)(dag ? j + 3 * i : i + 3 * j) * S];
      if (dag) x.im = -x.im;
      v[i + 3 * j] = x;
    }
  int top = 0, topd = 0;
  ll d[3], dor = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    top = max(top, habs(v[k].im));
    if (k % 4 == 0) {
      topd = max(topd, habs(v[k].re));
      const ll q = to_fixed(v[k].re, shift(kScale)) - (1LL << kScale);
      d[k / 4] = q;
      dor |= q ^ (q >> 63);
    } else {
      top = max(top, habs(v[k].re));
    }
  }
  g.bad |= max(top, topd) > kMaxEntryHi;
  constexpr int least = kMinExpOf<T>;
  const int ed = dor == 0 ? least : 64 - __clzll(dor) - kScale;  // |diagonal - 1| < 2^ed
  int ee = max(max(exponent_of(top), ed), least);
  if (sizeof(T) == 8) g.bad |= ee == least && top != 0;  // tiny
  ee = min(ee, 0);
  e = ee;
  const int kb = shift(kScale - ee);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    m.e[k].im = to_fixed_split(v[k].im, kb);
    m.e[k].re = k % 4 == 0 ? split(d[k / 4] << min(-ee, 63)) : to_fixed_split(v[k].re, kb);
  }
}

// ---- products -------------------------------------------------------------------------------------------
__device__ __forceinline__ R neg(const R& a) {
  R r;
  r.h = -a.h;
  r.l = -a.l;
  return r;
}
// (A B)_ij; nB: -Im of B's entries
__device__ __forceinline__ void entry_nn(const M& A, int i, const M& B, const R (&nB)[9], int j, Acc& re, Acc& im) {
  re = im = acc_half();
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const C &a = A.e[i + 3 * k], &b = B.e[k + 3 * j];
    mad(re, a.re, b.re);
    mad(re, a.im, nB[k + 3 * j]);
    mad(im, a.re, b.im);
    mad(im, a.im, b.re);
  }
}

// The rows of 1 + A must have norm one (to 10 %): looked at where an entry of A may reach 1/8.
__device__ __forceinline__ void unit_rows(const M& A, int e, Guard& g) {
  if (e < -2) return;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    ll n = 0;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const C& a = A.e[i + 3 * j];
      const int x = (a.re.h >> -e) + (i == j ? kOneH : 0), y = a.im.h >> -e;
      n += (ll)x * x + (ll)y * y;
    }
    const int t = (int)(n >> 32);  // 2^56 is one: 2^24 here
    g.bad |= n < 0 || t < (int)(0.81 * (1 << 24)) || t > (int)(1.21 * (1 << 24));
  }
}

// w = (1 + A)(1 + B) - 1, its exponent at most 0 and at least 3 above A's and B's (below the cap), so |w| < 2^e / 2
// there; at the cap |w| <= 2.
__device__ __forceinline__ void near_product(const M& A, int ea, const M& B, int eb, M& W, int& ew, Guard& g) {
  ew = min(max(ea, eb) + 3, 0);
  const int kk = min(ew - ea - eb, 63), ka = min(ew - ea, 63), kb = min(ew - eb, 63);
  R nB[9];
#pragma unroll
  for (int n = 0; n < 9; n++) nB[n] = neg(B.e[n].im);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      Acc re, im;
      entry_nn(A, i, B, nB, j, re, im);
      const C &a = A.e[i + 3 * j], &b = B.e[i + 3 * j];
      W.e[i + 3 * j].re = split((finish(re) >> kk) + (join(a.re) >> ka) + (join(b.re) >> kb));
      W.e[i + 3 * j].im = split((finish(im) >> kk) + (join(a.im) >> ka) + (join(b.im) >> kb));
    }
  if (ew == 0) unit_rows(W, 0, g);  // entries near or above 1/8
}

// The anti-Hermitian part of a matrix P: y_ij = Im(P_ij + P_ji), x_ij = Re(P_ij - P_ji) for (ij) = 01, 02, 12 and
// d_i = Im P_ii.  al = ReTr(i t P) is -1/2 of (y01, x01, d0 - d1, y02, x02, y12, x12, (d0 + d1 - 2 d2) / sqrt 3).
struct Anti {
  ll y[3], x[3], d[3];
  int e;
};
// component k of -2 al 2^(60-e), the last without its 1/sqrt(3)
__device__ __forceinline__ ll component(const Anti& p, int k) {
  switch (k) {
    case 0: return p.y[0];
    case 1: return p.x[0];
    case 2: return p.d[0] - p.d[1];
    case 3: return p.y[1];
    case 4: return p.x[1];
    case 5: return p.y[2];
    case 6: return p.x[2];
    default: return p.d[0] + p.d[1] - 2 * p.d[2];
  }
}

// P = (1 + w)(1 + v)^dagger of two near products
__device__ __forceinline__ void plaquette_parts(const M& W, int ew, const M& V, int ev, Anti& o) {
  const int ep = max(ew, ev);
  const int k = min(ep - ew - ev, 63), kw = min(ep - ew, 63), kv = min(ep - ev, 63);
  o.e = ep;
  constexpr int pi[3] = {0, 0, 1}, pj[3] = {1, 2, 2};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const int i = pi[n], j = pj[n];
    Acc yp = acc_half(), yn = acc_zero(), xp = acc_half(), xn = acc_zero();
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const C &wi = W.e[i + 3 * t], &wj = W.e[j + 3 * t], &vi = V.e[i + 3 * t], &vj = V.e[j + 3 * t];
      mad(yp, wi.im, vj.re);
      mad(yp, wj.im, vi.re);
      mad(yn, wi.re, vj.im);
      mad(yn, wj.re, vi.im);
      mad(xp, wi.re, vj.re);
      mad(xp, wi.im, vj.im);
      mad(xn, wj.re, vi.re);
      mad(xn, wj.im, vi.im);
    }
    o.y[n] = finish_diff(yp, yn) >> k;
    o.x[n] = finish_diff(xp, xn) >> k;
    const ll yw = join(W.e[i + 3 * j].im) + join(W.e[j + 3 * i].im), yv = join(V.e[i + 3 * j].im) + join(V.e[j + 3 * i].im);
    const ll xw = join(W.e[i + 3 * j].re) - join(W.e[j + 3 * i].re), xv = join(V.e[j + 3 * i].re) - join(V.e[i + 3 * j].re);
    o.y[n] += (yw >> kw) - (yv >> kv);
    o.x[n] += (xw >> kw) + (xv >> kv);
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    Acc p = acc_half(), q = acc_zero();
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const C &w = W.e[i + 3 * t], &v = V.e[i + 3 * t];
      mad(p, w.im, v.re);
      mad(q, w.re, v.im);
    }
    o.d[i] = (finish_diff(p, q) >> k) + (join(W.e[4 * i].im) >> kw) - (join(V.e[4 * i].im) >> kv);
  }
}

// -Re tr(P - 1) 2^(60-e), e = max(ew, ev), of the same P: 3 - Re tr P without its cancellation
__device__ __forceinline__ ll plaquette_trace(const M& W, int ew, const M& V, int ev) {
  const int ep = max(ew, ev);
  Acc a = acc_half();
#pragma unroll
  for (int k = 0; k < 9; k++) {
    mad(a, W.e[k].re, V.e[k].re);
    mad(a, W.e[k].im, V.e[k].im);
  }
  const ll w = join(W.e[0].re) + join(W.e[4].re) + join(W.e[8].re), v = join(V.e[0].re) + join(V.e[4].re) + join(V.e[8].re);
  return -((finish(a) >> min(ep - ew - ev, 63)) + (w >> min(ep - ew, 63)) + (v >> min(ep - ev, 63)));
}

// M = H(p) + i H(q) with H_ij = y_ij - i x_ij, H_ji its conjugate (i < j), H_ii = 2 d_i - 2/3 sum d: H(p) = -4 t.al.
// Exponent e; the two exponents may differ.
__device__ __forceinline__ void herm_pair(const Anti& p, const Anti& q, M& m, int& e) {
  const int em = max(p.e, q.e) + 1;
  const int kp = min(em - p.e, 63), kq = min(em - q.e, 63);
  e = em;
  constexpr int pi[3] = {0, 0, 1}, pj[3] = {1, 2, 2};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const int i = pi[n], j = pj[n];
    const ll y1 = p.y[n] >> kp, x1 = p.x[n] >> kp, y2 = q.y[n] >> kq, x2 = q.x[n] >> kq;
    m.e[i + 3 * j].re = split(y1 + x2);
    m.e[i + 3 * j].im = split(y2 - x1);
    m.e[j + 3 * i].re = split(y1 - x2);
    m.e[j + 3 * i].im = split(y2 + x1);
  }
  constexpr ll third = 0x5555555555555556LL;
  const ll tp = __mul64hi(p.d[0] + p.d[1] + p.d[2], third), tq = __mul64hi(q.d[0] + q.d[1] + q.d[2], third);
  const ll a0 = (p.d[0] - tp) >> (kp - 1), a1 = (p.d[1] - tp) >> (kp - 1);
  const ll b0 = (q.d[0] - tq) >> (kq - 1), b1 = (q.d[1] - tq) >> (kq - 1);
  m.e[0].re = split(a0);
  m.e[0].im = split(b0);
  m.e[4].re = split(a1);
  m.e[4].im = split(b1);
  m.e[8].re = split(-a0 - a1);
  m.e[8].im = split(-b0 - b1);
}

// Sums of watched numbers (below 4 each) that may pass the format's 8, from their high words (2^28 is one): 3 (a + b), and
// a + b - 2 c.  Links of SU(3) stay far below; a matrix with large entries that is not unitary need not.
__device__ __forceinline__ void watch_sum(Guard& g, ll a, ll b) {
  constexpr unsigned most = 5u << 27;  // 2.5
  g.bad |= (unsigned)((int)(a >> 32) + (int)(b >> 32)) + most > 2 * most;
}
__device__ __forceinline__ void watch_eighth(Guard& g, ll a, ll b, ll c) {
  constexpr int most = 15 << 25;  // 7.5 / 4
  g.bad |= abs((int)(a >> 34) + (int)(b >> 34) - (int)(c >> 33)) > most;
}

// The Hermitian and anti-Hermitian parts of C = V^dagger M V (kInv) or V M V^dagger, as split_herm_pair gives them
// (the last of each without its 1/sqrt(3)); V plain, in units of M.  M is traceless, and C_22 follows from that.
template <bool kInv>
__device__ __forceinline__ void rotate_pair(const M& V, const M& Mm, ll (&o1)[8], ll (&o2)[8], Guard& g) {
  ll cr[9], ci[9];
  R nV[9];
#pragma unroll
  for (int n = 0; n < 9; n++) nV[n] = neg(V.e[n].im);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    C t[3];  // row i of V^dagger M, or of V M
#pragma unroll
    for (int j = 0; j < 3; j++) {
      Acc re = acc_half(), im = acc_half();
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const C& m = Mm.e[k + 3 * j];
        const int n = kInv ? k + 3 * i : i + 3 * k;  // conj(v) m or v m
        mad(re, V.e[n].re, m.re);
        mad(re, kInv ? V.e[n].im : nV[n], m.im);
        mad(im, V.e[n].re, m.im);
        mad(im, kInv ? nV[n] : V.e[n].im, m.re);
      }
      watch(g, re.hh, im.hh);
      t[j].re = split(finish(re));
      t[j].im = split(finish(im));
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
      if (i == 2 && j == 2) continue;
      Acc re = acc_half(), im = acc_half();
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int n = kInv ? k + 3 * j : j + 3 * k;  // t v or t conj(v)
        mad(re, t[k].re, V.e[n].re);
        mad(re, t[k].im, kInv ? nV[n] : V.e[n].im);
        mad(im, t[k].im, V.e[n].re);
        mad(im, t[k].re, kInv ? V.e[n].im : nV[n]);
      }
      watch(g, re.hh, im.hh);
      cr[i + 3 * j] = finish(re);
      ci[i + 3 * j] = finish(im);
    }
  }
  watch_sum(g, cr[0], cr[4]);
  watch_sum(g, ci[0], ci[4]);
  o1[0] = cr[3] + cr[1];
  o1[1] = ci[1] - ci[3];
  o1[2] = cr[0] - cr[4];
  o1[3] = cr[6] + cr[2];
  o1[4] = ci[2] - ci[6];
  o1[5] = cr[7] + cr[5];
  o1[6] = ci[5] - ci[7];
  o1[7] = 3 * (cr[0] + cr[4]);
  o2[0] = ci[3] + ci[1];
  o2[1] = cr[3] - cr[1];
  o2[2] = ci[0] - ci[4];
  o2[3] = ci[6] + ci[2];
  o2[4] = cr[6] - cr[2];
  o2[5] = ci[7] + ci[5];
  o2[6] = cr[7] - cr[5];
  o2[7] = 3 * (ci[0] + ci[4]);
}

// C = V^dagger H V for Hermitian H, as alg_from_herm reads it (the last component without its 1/sqrt(3), all doubled as
// in rotate_pair): the upper triangle of C and its diagonal.  (C_22 is formed, not taken from the trace: that is zero
// only as far as V is unitary, which on links built as long products shows at 1e-15.)
__device__ __forceinline__ void rotate_one(const M& V, const M& H, ll (&o)[8], Guard& g) {
  ll cr[9], ci[9];
  R nV[9];
#pragma unroll
  for (int n = 0; n < 9; n++) nV[n] = neg(V.e[n].im);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    C t[3];  // row i of V^dagger H; H_jj is real
#pragma unroll
    for (int j = 0; j < 3; j++) {
      Acc re = acc_half(), im = acc_half();
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const C& m = H.e[k + 3 * j];
        const int n = k + 3 * i;
        mad(re, V.e[n].re, m.re);
        mad(im, nV[n], m.re);
        if (k != j) {
          mad(re, V.e[n].im, m.im);
          mad(im, V.e[n].re, m.im);
        }
      }
      watch(g, re.hh, im.hh);
      t[j].re = split(finish(re));
      t[j].im = split(finish(im));
    }
#pragma unroll
    for (int j = i; j < 3; j++) {
      Acc re = acc_half(), im = acc_half();
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int n = k + 3 * j;
        mad(re, t[k].re, V.e[n].re);
        mad(re, t[k].im, nV[n]);
        if (j != i) {
          mad(im, t[k].im, V.e[n].re);
          mad(im, t[k].re, V.e[n].im);
        }
      }
      watch(g, re.hh, im.hh);
      cr[i + 3 * j] = finish(re);
      ci[i + 3 * j] = finish(im);
    }
  }
  watch_eighth(g, cr[0], cr[4], cr[8]);
  o[0] = 2 * cr[3];
  o[1] = -2 * ci[3];
  o[2] = cr[0] - cr[4];
  o[3] = 2 * cr[6];
  o[4] = -2 * ci[6];
  o[5] = 2 * cr[7];
  o[6] = -2 * ci[7];
  o[7] = cr[0] + cr[4] - 2 * cr[8];
}
// 2 t.p
template <typename T>
__device__ __forceinline__ void herm_one(const Alg<T>& p, M& m, int& e, Guard& g) {
  int top = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) top = max(top, habs(p.a[k]));
  g.bad |= top >= 0x43100000 || (sizeof(T) == 8 && tiny(top));  // 2^50 or more, or not finite
  const int em = max(exponent_of(min(top, 0x43100000)), kMinExpOf<T>) + 2;
  e = em;
  const int sh = shift(kScale - em);
  // a_8 / sqrt 3 in FP64: exact in the format to 2^-60 whatever T is
  const ll s8 = to_fixed((double)p.a[7] * Consts<double>::inv_sqrt3(), sh), c = to_fixed(p.a[2], sh);
  constexpr int pi[3] = {0, 0, 1}, pj[3] = {1, 2, 2}, py[3] = {0, 3, 5};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const int u = pi[n] + 3 * pj[n], l = pj[n] + 3 * pi[n];
    m.e[u].re = m.e[l].re = to_fixed_split(p.a[py[n]], sh);
    m.e[l].im = to_fixed_split(p.a[py[n] + 1], sh);
    m.e[u].im = neg(m.e[l].im);
  }
  m.e[0].re = split(c + s8);
  m.e[4].re = split(s8 - c);
  m.e[8].re = split(-2 * s8);
}

// M = 2 (t.p + i t.q) from two FP64 algebra vectors, exponent two above their largest component's.
__device__ __forceinline__ void herm_pair(const Alg<double>& p, const Alg<double>& q, M& m, int& e, Guard& g) {
  int top = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) top = max(top, max(habs(p.a[k]), habs(q.a[k])));
  g.bad |= top >= 0x43100000 || tiny(top);  // 2^50 or more, or not finite
  const int em = max(exponent_of(min(top, 0x43100000)), kMinExp) + 2;
  e = em;
  const int kb = shift(kScale - em);
  const ll s1 = to_fixed(p.a[7] * Consts<double>::inv_sqrt3(), kb), s2 = to_fixed(q.a[7] * Consts<double>::inv_sqrt3(), kb);
  constexpr int pi[3] = {0, 0, 1}, pj[3] = {1, 2, 2}, py[3] = {0, 3, 5};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const int i = pi[n], j = pj[n];
    const ll y1 = to_fixed(p.a[py[n]], kb), x1 = to_fixed(p.a[py[n] + 1], kb);
    const ll y2 = to_fixed(q.a[py[n]], kb), x2 = to_fixed(q.a[py[n] + 1], kb);
    m.e[i + 3 * j].re = split(y1 + x2);
    m.e[i + 3 * j].im = split(y2 - x1);
    m.e[j + 3 * i].re = split(y1 - x2);
    m.e[j + 3 * i].im = split(y2 + x1);
  }
  const ll c1 = to_fixed(p.a[2], kb), c2 = to_fixed(q.a[2], kb);
  m.e[0].re = split(c1 + s1);
  m.e[0].im = split(c2 + s2);
  m.e[4].re = split(s1 - c1);
  m.e[4].im = split(s2 - c2);
  m.e[8].re = split(-2 * s1);
  m.e[8].im = split(-2 * s2);
}

// +-2^k o, the last component over sqrt 3; kFp64: by the FP64 pipe
template <bool kFp64 = false>
__device__ __forceinline__ void to_alg(const ll (&o)[8], int k, double sign, Alg<double>& out) {
#pragma unroll
  for (int n = 0; n < 8; n++) {
    const double v = kFp64 ? from_fixed_fp64(o[n], k) : from_fixed(o[n], k);
    out.a[n] = n == 7 ? v * (sign * Consts<double>::inv_sqrt3()) : (sign < 0 ? -v : v);
  }
}

// Two adjoint actions by one plain matrix, as inv_adj_mul2 / adj_mul2: out_k = V^d (t.e_k) V or V (t.e_k) V^d.
template <bool kInv>
__device__ __forceinline__ void adj_pair(const M& V, const Alg<double>& e1, const Alg<double>& e2, Alg<double>& out1,
                                         Alg<double>& out2, Guard& g) {
  M m;
  int e;
  ll o1[8], o2[8];
  herm_pair(e1, e2, m, e, g);
  rotate_pair<kInv>(V, m, o1, o2, g);
  to_alg(o1, e - kScale - 1, 1.0, out1);
  to_alg(o2, e - kScale - 1, 1.0, out2);
}


// A matrix of doubles with the exponent of its largest entry; kLink: exponent 0 and entries up to one (1.03).
template <bool kLink>
__device__ __forceinline__ void from_mat(const Mat<double>& u, M& m, int& e, Guard& g) {
  int top = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) top = max(top, max(habs(u.e[k].re), habs(u.e[k].im)));
  g.bad |= kLink ? top > kMaxEntryHi : top >= 0x43100000;
  e = kLink ? 0 : max(exponent_of(min(top, 0x43100000)), kMinExp);
  const int kb = shift(kScale - e);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    m.e[k].re = to_fixed_split(u.e[k].re, kb);
    m.e[k].im = to_fixed_split(u.e[k].im, kb);
  }
}

// ---- the link update's exponential -----------------------------------------------------------------------
// f0 - 1, f1, f2 of exp(iQ) = f0 + f1 Q + f2 Q^2 for c1 = tr Q^2 / 2 >= 0.02 (expi_impl's tiers), out of line.
static __device__ __noinline__ void exp_coefficients(double c0, double c1, double (&f)[6]) {
  cx<double> f0, f1, f2;
  exp_coeff<double, true>(c0, c1, f0, f1, f2);
  f[0] = f0.re;
  f[1] = f0.im;
  f[2] = f1.re;
  f[3] = f1.im;
  f[4] = f2.re;
  f[5] = f2.im;
}

// X - 1 = exp(i c t.al) - 1 in fixed point, exponent e.  False when |c al| has a component of one or more.
// With B = 2 Q (entries of c al without the factors 1/2) in units of 2^em, em one above the largest component's
// exponent: Q^2 = B^2 / 4, c1 = tr B^2 / 8, det Q = det B / 8 from 28 products; c0 and c1 leave as doubles, and below
// c1 = 0.02 (c al up to ~0.1 in every component) f0 - 1, f1, f2 are polynomials in them, exp's power series reduced by
// Q^3 = c1 Q + c0 and cut after Q^11 / 11! (the next term is below 7e-19): 34 FP64 operations, where the
// matrix form of this exponential takes ~150.
__device__ __forceinline__ bool near_exp(double c, const Alg<double>& al, M& X, int& e) {
  Alg<double> q;
  int top = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    q.a[k] = c * al.a[k];
    top = max(top, habs(q.a[k]));
  }
  if (top >= 0x3ff00000 || tiny(top)) return false;  // also NaN and infinity
  const int em = max(exponent_of(top), kMinExp) + 1;
  const int sh = shift(kScale - em);
  const ll s8 = to_fixed(q.a[7] * Consts<double>::inv_sqrt3(), sh), q2 = to_fixed(q.a[2], sh);
  R b[3];  // diagonal of B
  C o[3];  // B_01, B_02, B_12
  b[0] = split(q2 + s8);
  b[1] = split(s8 - q2);
  b[2] = split(-2 * s8);
  constexpr int comp[3] = {0, 3, 5};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    o[n].re = to_fixed_split(q.a[comp[n]], sh);
    o[n].im = to_fixed_split(-q.a[comp[n] + 1], sh);
  }
  // moduli, products of two off-diagonal entries
  ll mod[3];
#pragma unroll
  for (int n = 0; n < 3; n++) {
    Acc a = acc_half();
    mad(a, o[n].re, o[n].re);
    mad(a, o[n].im, o[n].im);
    mod[n] = finish(a);
  }
  auto product = [&](const C& u, const C& v, int conj_of, ll& re, ll& im) {  // conj_of: 0 none, 1 of u, 2 of v
    Acc a = acc_half(), z = acc_half(), y = acc_zero();
    if (conj_of == 0) {  // (ur vr - ui vi, ur vi + ui vr)
      mad(z, u.re, v.re);
      mad(y, u.im, v.im);
      mad(a, u.re, v.im);
      mad(a, u.im, v.re);
      re = finish_diff(z, y);
      im = finish(a);
    } else {  // (ur vr + ui vi, +-(ur vi - ui vr))
      mad(a, u.re, v.re);
      mad(a, u.im, v.im);
      mad(z, conj_of == 1 ? u.re : u.im, conj_of == 1 ? v.im : v.re);
      mad(y, conj_of == 1 ? u.im : u.re, conj_of == 1 ? v.re : v.im);
      re = finish(a);
      im = finish_diff(z, y);
    }
  };
  auto times = [&](const R& u, const R& v) {
    Acc a = acc_half();
    mad(a, u, v);
    return finish(a);
  };
  ll pr[3], pi[3];
  product(o[1], o[2], 2, pr[0], pi[0]);  // B02 conj(B12)
  product(o[0], o[2], 0, pr[1], pi[1]);  // B01 B12
  product(o[0], o[1], 1, pr[2], pi[2]);  // conj(B01) B02
  ll det = 0;
  {
    C t;
    t.re = split(pr[1]);
    t.im = split(pi[1]);
    const R n = split(times(b[1], b[2]) - mod[2]);
    Acc a = acc_half(), d = acc_zero();
    mad(a, t.re, o[1].re);
    mad(a, t.im, o[1].im);
    det = 2 * finish(a);
    a = acc_half();
    mad(a, b[0], n);
    mad(d, b[1], split(mod[1]));
    mad(d, b[2], split(mod[0]));
    det += finish_diff(a, d);
  }
  const ll d0 = times(b[0], b[0]) + mod[0] + mod[1], d1 = times(b[1], b[1]) + mod[0] + mod[2],
           d2 = times(b[2], b[2]) + mod[1] + mod[2];
  // below 2^-100 both are lost next to one (and the exponent of det would leave the doubles' range)
  const bool weak = em < -100;
  const double c1 = weak ? 0.0 : from_fixed(d0 + d1 + d2, 2 * em - kScale - 3);
  const double c0 = weak ? 0.0 : from_fixed(det, 3 * em - kScale - 3);
  double f[6];
  if (c1 < 0.02) {
    const double z = c0 * c0;
    f[0] = z * fma(c1, fma(c1, -1.0 / 1209600, 1.0 / 20160), -1.0 / 720);
    f[1] = c0 * fma(z, 1.0 / 362880, fma(c1, fma(c1, fma(c1, fma(c1, -1.0 / 39916800, 1.0 / 362880), -1.0 / 5040), 1.0 / 120), -1.0 / 6));
    f[2] = c0 * fma(z, -1.0 / 3628800, fma(c1, fma(c1, fma(c1, -1.0 / 907200, 1.0 / 13440), -1.0 / 360), 1.0 / 24));
    f[3] = fma(z, fma(c1, fma(c1, -1.0 / 6652800, 1.0 / 120960), -1.0 / 5040),
               fma(c1, fma(c1, fma(c1, fma(c1, fma(c1, -1.0 / 39916800, 1.0 / 362880), -1.0 / 5040), 1.0 / 120), -1.0 / 6), 1.0));
    f[4] = fma(z, fma(c1, -1.0 / 1209600, 1.0 / 40320),
               fma(c1, fma(c1, fma(c1, fma(c1, -1.0 / 3628800, 1.0 / 40320), -1.0 / 720), 1.0 / 24), -0.5));
    f[5] = c0 * fma(z, -1.0 / 39916800, fma(c1, fma(c1, fma(c1, -1.0 / 9979200, 1.0 / 120960), -1.0 / 2520), 1.0 / 120));
  } else {
    exp_coefficients(c0, c1, f);
  }
  // X - 1 = f0 - 1 + (f1 B + 2^(em-1) (f2 / 2^(em-1)) B^2 / 2) / 2 in units of 2^(em-1): B^2 moved to B's units
  e = em - 1;
  const int down = min(1 - em, 63);
  C g1, g2;
  g1.re = to_fixed_split(f[2], shift(kScale));
  g1.im = to_fixed_split(f[3], shift(kScale));
  g2.re = to_fixed_split(f[4], shift(kScale));
  g2.im = to_fixed_split(f[5], shift(kScale));
  constexpr int up[3] = {3, 6, 7}, low[3] = {1, 2, 5}, opp[3] = {2, 1, 0};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    C w;  // (B^2)_ij = -B_kk B_ij + B_ik B_kj
    w.re = split((pr[n] - times(b[opp[n]], o[n].re)) >> down);
    w.im = split((pi[n] - times(b[opp[n]], o[n].im)) >> down);
    Acc r = acc_half(), s = acc_half(), t = acc_half(), u = acc_half();
    mad(r, g1.re, o[n].re);
    mad(r, g2.re, w.re);
    mad(s, g1.im, o[n].im);
    mad(s, g2.im, w.im);
    mad(t, g1.re, o[n].im);
    mad(t, g2.re, w.im);
    mad(u, g1.im, o[n].re);
    mad(u, g2.im, w.re);
    const ll rr = finish(r), ss = finish(s), tt = finish(t), uu = finish(u);
    X.e[up[n]].re = split(rr - ss);
    X.e[up[n]].im = split(uu + tt);
    X.e[low[n]].re = split(rr + ss);
    X.e[low[n]].im = split(uu - tt);
  }
  const ll f0r = to_fixed(f[0], shift(kScale - e)), f0i = to_fixed(f[1], shift(kScale - e));
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const R w = split((n == 0 ? d0 : (n == 1 ? d1 : d2)) >> down);
    Acc r = acc_half(), u = acc_half();
    mad(r, g1.re, b[n]);
    mad(r, g2.re, w);
    mad(u, g1.im, b[n]);
    mad(u, g2.im, w);
    X.e[4 * n].re = split(finish(r) + f0r);
    X.e[4 * n].im = split(finish(u) + f0i);
  }
  return true;
}

// out = u + A u for A = X - 1 in fixed point and a link u: the product with A's exponent, the sum in FP64, so the
// result is rounded once.  False where the format does not hold u.
__device__ __forceinline__ bool add_product(const M& a, int ea, const Mat<double>& u, Mat<double>& out) {
  Guard g = guard_init();
  M b;
  int eb;
  from_mat<true>(u, b, eb, g);
  R nb[9];
#pragma unroll
  for (int n = 0; n < 9; n++) nb[n] = neg(b.e[n].im);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      Acc re, im;
      entry_nn(a, i, b, nb, j, re, im);
      out.e[i + 3 * j].re = u.e[i + 3 * j].re + from_fixed(finish(re), ea - kScale);
      out.e[i + 3 * j].im = u.e[i + 3 * j].im + from_fixed(finish(im), ea - kScale);
    }
  return !g.bad;
}

// P - 1 of P = (1 + w)(1 + v)^dagger in full: its anti-Hermitian part, and the Hermitian part h of P - 1 as doubles
// (h_ij, i <= j).
__device__ __forceinline__ void plaquette_full(const M& W, int ew, const M& V, int ev, Anti& o, Mat<double>& h) {
  const int ep = max(ew, ev);
  const int k = min(ep - ew - ev, 63), kw = min(ep - ew, 63), kv = min(ep - ev, 63);
  o.e = ep;
  R nV[9];
#pragma unroll
  for (int n = 0; n < 9; n++) nV[n] = neg(V.e[n].im);
  auto entry = [&](int i, int j, ll& re, ll& im) {
    Acc a = acc_half(), b = acc_half();
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const C& w = W.e[i + 3 * t];
      mad(a, w.re, V.e[j + 3 * t].re);
      mad(a, w.im, V.e[j + 3 * t].im);
      mad(b, w.im, V.e[j + 3 * t].re);
      mad(b, w.re, nV[j + 3 * t]);
    }
    re = (finish(a) >> k) + (join(W.e[i + 3 * j].re) >> kw) + (join(V.e[j + 3 * i].re) >> kv);
    im = (finish(b) >> k) + (join(W.e[i + 3 * j].im) >> kw) - (join(V.e[j + 3 * i].im) >> kv);
  };
  constexpr int pi[3] = {0, 0, 1}, pj[3] = {1, 2, 2};
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const int i = pi[n], j = pj[n];
    ll ru, iu, rl, il;
    entry(i, j, ru, iu);
    entry(j, i, rl, il);
    o.y[n] = iu + il;
    o.x[n] = ru - rl;
    h.e[i + 3 * j] = mk<double>(from_fixed(ru + rl, ep - kScale - 1), from_fixed(iu - il, ep - kScale - 1));
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    ll r, m;
    entry(i, i, r, m);
    o.d[i] = m;
    h.e[4 * i] = mk<double>(from_fixed(r, ep - kScale), 0.0);
  }
}

// The structure-constant product c = q x t (c^k = f^klm q_l t_m) of two vectors whose eighth components carry a factor
// sqrt 3, as c's does: every constant but f^123 is 1/2 then.
__device__ __forceinline__ void cross8(const R (&Q)[8], const R (&T)[8], ll (&c)[8]) {
  R N[8];
#pragma unroll
  for (int k = 0; k < 8; k++) N[k] = neg(T[k]);
  auto d = [&](Acc& a, int i, int j) {  // Q_i T_j - Q_j T_i
    mad(a, Q[i - 1], T[j - 1]);
    mad(a, Q[j - 1], N[i - 1]);
  };
  Acc a = acc_half(), b = acc_half();
  d(a, 2, 3), d(b, 4, 7), d(b, 6, 5);
  c[0] = finish(a) + (finish(b) >> 1);
  a = b = acc_half();
  d(a, 3, 1), d(b, 4, 6), d(b, 5, 7);
  c[1] = finish(a) + (finish(b) >> 1);
  a = b = acc_half();
  d(a, 1, 2), d(b, 4, 5), d(b, 7, 6);
  c[2] = finish(a) + (finish(b) >> 1);
  a = acc_half();
  d(a, 7, 1), d(a, 6, 2), d(a, 5, 3), d(a, 5, 8);
  c[3] = finish(a) >> 1;
  a = acc_half();
  d(a, 1, 6), d(a, 7, 2), d(a, 3, 4), d(a, 8, 4);
  c[4] = finish(a) >> 1;
  a = acc_half();
  d(a, 5, 1), d(a, 2, 4), d(a, 3, 7), d(a, 7, 8);
  c[5] = finish(a) >> 1;
  a = acc_half();
  d(a, 1, 4), d(a, 2, 5), d(a, 6, 3), d(a, 8, 6);
  c[6] = finish(a) >> 1;
  a = acc_half();
  d(a, 4, 5), d(a, 6, 7);
  const ll r = finish(a);
  c[7] = r + (r >> 1);
}
constexpr double kRoot3 = 1.7320508075688772935;
// the larger |high word| of a vector's components, the eighth times sqrt 3
__device__ __forceinline__ int top_of(const Alg<double>& v, double v8) {
  int t = habs(v8);
#pragma unroll
  for (int k = 0; k < 7; k++) t = max(t, habs(v.a[k]));
  return t;
}
// its components below 2^(60-e) |v| < 2^60
__device__ __forceinline__ void to_fixed_alg(const Alg<double>& v, double v8, int e, R (&o)[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) o[k] = to_fixed_split(k == 7 ? v8 : v.a[k], shift(kScale - e));
}
constexpr int kMaxHi = 0x43100000;  // 2^50

// out = a x b; false where the format does not hold the operands
__device__ __forceinline__ bool cross(const Alg<double>& a, const Alg<double>& b, Alg<double>& out) {
  const double a8 = a.a[7] * kRoot3, b8 = b.a[7] * kRoot3;
  const int ta = top_of(a, a8), tb = top_of(b, b8);
  if (max(ta, tb) >= kMaxHi || tiny<true>(ta) || tiny<true>(tb)) return false;  // the product's exponent is the sum
  const int ea = max(exponent_of(ta), kMinExp / 2), eb = max(exponent_of(tb), kMinExp / 2) + 1;
  R A[8], B[8];
  ll c[8];
  to_fixed_alg(a, a8, ea, A);
  to_fixed_alg(b, b8, eb, B);
  cross8(A, B, c);
#pragma unroll
  for (int k = 0; k < 8; k++) out.a[k] = from_fixed(c[k], ea + eb - kScale) * (k == 7 ? kRoot3 / 3 : 1.0);
  return true;
}

// out^k = Re tr(t^k H t.n) = 1/4 Re tr(t^k {H, 2 t.n}) for Hermitian H (h_ii, and h_ij for i < j)
__device__ __forceinline__ bool trace_with(const Mat<double>& h, const Alg<double>& n, Alg<double>& out) {
  const double n8 = n.a[7] * Consts<double>::inv_sqrt3();
  int th = 0, tn = top_of(n, n8);
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int i = 0; i <= j; i++) th = max(th, max(habs(h.e[i + 3 * j].re), habs(h.e[i + 3 * j].im)));
  if (max(th, tn) >= kMaxHi || tiny<true>(th) || tiny<true>(tn)) return false;
  // sums of two diagonal entries stay below 1, those of 2 t.n (up to 1.16 of the components) below 1 too
  const int eh = max(exponent_of(th), kMinExp / 2) + 1, en = max(exponent_of(tn), kMinExp / 2) + 2;
  const int sh = shift(kScale - eh), sn = shift(kScale - en);
  ll hd[3], bd[3];
  C ho[3], bo[3];  // 01, 02, 12
  constexpr int at[3] = {3, 6, 7}, comp[3] = {0, 3, 5};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    hd[k] = to_fixed(h.e[4 * k].re, sh);
    ho[k].re = to_fixed_split(h.e[at[k]].re, sh);
    ho[k].im = to_fixed_split(h.e[at[k]].im, sh);
    bo[k].re = to_fixed_split(n.a[comp[k]], sn);
    bo[k].im = to_fixed_split(-n.a[comp[k] + 1], sn);
  }
  const ll b3 = to_fixed(n.a[2], sn), b8 = to_fixed(n8, sn);
  bd[0] = b8 + b3;
  bd[1] = b8 - b3;
  bd[2] = -2 * b8;
  // the diagonal: h_i b_i and r_n = Re(h_n conj(b_n))
  ll hb[3], r[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    Acc a = acc_half(), b = acc_half();
    mad(a, split(hd[k]), split(bd[k]));
    mad(b, ho[k].re, bo[k].re);
    mad(b, ho[k].im, bo[k].im);
    hb[k] = finish(a);
    r[k] = finish(b);
  }
  // off the diagonal: (h_i + h_j) b_n + (b_i + b_j) h_n + u v + w x, with the conjugates the indices ask for
  ll re[3], im[3];
  auto off = [&](int n_, int i, int j, const C& u, int su, const C& v, int sv, const C& w, int sw, const C& x, int sx) {
    Acc a = acc_half(), b = acc_half();
    const R hh = split(hd[i] + hd[j]), bb = split(bd[i] + bd[j]);
    mad(a, hh, bo[n_].re);
    mad(b, hh, bo[n_].im);
    mad(a, bb, ho[n_].re);
    mad(b, bb, ho[n_].im);
    auto times = [&](const C& p, int sp, const C& q, int sq) {
      const R pi = sp < 0 ? neg(p.im) : p.im, qi = sq < 0 ? neg(q.im) : q.im;
      mad(a, p.re, q.re);
      mad(a, neg(pi), qi);
      mad(b, p.re, qi);
      mad(b, pi, q.re);
    };
    times(u, su, v, sv);
    times(w, sw, x, sx);
    re[n_] = finish(a);
    im[n_] = finish(b);
  };
  off(0, 0, 1, ho[1], 1, bo[2], -1, bo[1], 1, ho[2], -1);
  off(1, 0, 2, ho[0], 1, bo[2], 1, bo[0], 1, ho[2], 1);
  off(2, 1, 2, ho[0], -1, bo[1], 1, bo[0], -1, ho[1], 1);
  const int k = eh + en - kScale;
#pragma unroll
  for (int m = 0; m < 3; m++) {
    out.a[comp[m]] = from_fixed(re[m], k - 2);
    out.a[comp[m] + 1] = -from_fixed(im[m], k - 2);
  }
  out.a[2] = from_fixed((hb[0] - hb[1]) + (r[1] - r[2]), k - 2);
  out.a[7] = from_fixed((hb[0] + hb[1] - 2 * hb[2]) + (2 * r[0] - r[1] - r[2]), k - 2) * Consts<double>::inv_sqrt3();
  return true;
}

// sum_n (q x)^n l / (n + 1)! in fixed point, n up to `terms`; inv[n] = 1 / n.  The caller has |q| < 1 (as a vector), so no term
// is larger than l and the sum below 2 |l|; a component of q, the eighth times sqrt 3, then stays below 2.
__device__ __forceinline__ bool exp_series(const Alg<double>& q, const Alg<double>& l, int terms, const double* inv,
                                           Alg<double>& out) {
  const double q8 = q.a[7] * kRoot3, l8 = l.a[7] * kRoot3;
  const int tq = top_of(q, q8), tl = top_of(l, l8);
  if (tq >= 0x40000000 || tl >= kMaxHi || tiny(tl)) return false;  // 2
  const int eq = max(exponent_of(tq), kMinExp), el = max(exponent_of(tl), kMinExp) + 1;
  const int down = min(-min(eq, 0), 63), up = max(eq, 0);
  R Q[8], T[8];
  ll sum[8];
  to_fixed_alg(q, q8, eq, Q);
  to_fixed_alg(l, l8, el, T);
#pragma unroll
  for (int k = 0; k < 8; k++) sum[k] = join(T[k]);
#pragma unroll 1
  for (int n = 1; n <= terms; n++) {
    ll c[8];
    cross8(Q, T, c);
    const R f = to_fixed_split(inv[n + 1], shift(kScale));
#pragma unroll
    for (int k = 0; k < 8; k++) {
      Acc a = acc_half();
      mad(a, split((c[k] >> down) << up), f);
      const ll t = finish(a);
      T[k] = split(t);
      sum[k] += t;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; k++) out.a[k] = from_fixed(sum[k], el - kScale) * (k == 7 ? kRoot3 / 3 : 1.0);
  return true;
}

}  // namespace fx
}  // namespace glasma
