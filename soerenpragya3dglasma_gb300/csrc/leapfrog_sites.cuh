// leapfrog_sites.cuh -- per-site bodies of the two leapfrog kernels, shared by the single-lattice
// launches (leapfrog.cu) and the batched multi-event launches (batch.cu).
#pragma once

#include "fx.cuh"
#include "lattice.cuh"

namespace glasma {


constexpr int kThreads = 128;

// Pairs of adjoint actions by one matrix go through inv_adj_mul2 / adj_mul2 (one product pair instead
// of two); the double-float force kernel keeps its out-of-line single actions (ddf.cuh).
template <typename TC>
constexpr bool kPairRotations = !std::is_same<TC, ddf>::value;
// The pairs of the current transport (Jp and Jm rotated by one link) only in FP64: at the FP32 link kernels'
// 64-register cap the paired form spills.
template <typename T>
constexpr bool kPairCurrents = std::is_same<T, double>::value;

// What the integer pipe's fixed-point products hand back (fx.cuh), out of line.
template <bool adj>
__device__ __noinline__ void rotate_pair_fp64(const Mat<double>& V, const Alg<double>& ep, const Alg<double>& em,
                                              Alg<double>& out_p, Alg<double>& out_m) {
  if constexpr (adj)
    adj_mul2(V, ep, em, out_p, out_m);
  else
    inv_adj_mul2(V, ep, em, out_p, out_m);
}
static __device__ __noinline__ void link_step_fp64(double c, const Alg<double>& e, const Mat<double>& u,
                                                  Mat<double>& out) {
  Mat<double> X;
  link_exp(c, e, X);
  mul_near_identity(X, u, out);
}

// out_p = V (t.ep) V^d, out_m = V (t.em) V^d (adj = true) or the V^d . V forms, paired where kPairCurrents, in FP64 on
// the integer pipe
template <typename T, bool adj>
__device__ __forceinline__ void rotate_currents(const Mat<T>& V, const Alg<T>& ep, const Alg<T>& em, Alg<T>& out_p,
                                                Alg<T>& out_m) {
  if constexpr (kPairCurrents<T>) {
    fx::Guard g = fx::guard_init();
    fx::M v;
    int e;
    fx::from_mat<true>(V, v, e, g);
    fx::adj_pair<!adj>(v, ep, em, out_p, out_m, g);
    if (fx::tripped(g)) {
      const Mat<double> Vc = V;
      const Alg<double> a = ep, b = em;
      Alg<double> oa, ob;
      rotate_pair_fp64<adj>(Vc, a, b, oa, ob);
      out_p = oa;
      out_m = ob;
    }
  } else {
    if constexpr (adj) {
      adj_mul(V, ep, out_p);
      adj_mul(V, em, out_m);
    } else {
      inv_adj_mul(V, ep, out_p);
      inv_adj_mul(V, em, out_m);
    }
  }
}

// The link update u -> exp(i c t.e) u: the exponential formed once, applied once or twice.  FP32 as mul_near_identity,
// FP64 in fixed point on the integer pipe (fx.cuh), or in FP64 where that does not hold the numbers.
template <typename T>
struct LinkStep {
  Mat<T> X;
  __device__ __forceinline__ void set(T c, const Alg<T>& e) { link_exp(c, e, X); }
  __device__ __forceinline__ void apply(const Mat<T>& u, Mat<T>& out) const { mul_near_identity(X, u, out); }
};
template <>
struct LinkStep<double> {
  fx::M X;
  int ex;
  bool ok;
  double c;
  Alg<double> e;
  __device__ __forceinline__ void set(double c_, const Alg<double>& e_) {
    c = c_;
    e = e_;
    ex = 0;
    ok = fx::near_exp(c, e, X, ex);
  }
  __device__ __forceinline__ void apply(const Mat<double>& u, Mat<double>& out) const {
    Mat<double> o;
    if (!ok || !fx::add_product(X, ex, u, o)) {
      const Mat<double> b = u;
      const Alg<double> a = e;
      link_step_fp64(c, a, b, o);
    }
    out = o;
  }
};

// Blocks per SM the register allocation must leave room for (the register cap is 64K / (128 * n)),
// chosen by measurement on GB300; overridable at build time for tuning sweeps.
// (GB300 sweep, 128x128x512: FP32 K1 fastest at 5 blocks/SM, K2 at 8; the staple kernels in FP64 are FP64-ALU bound.
// The fixed-point kernels: force 10.9 ms at 3 blocks/SM, 12.4 at 2, 12.6 at 4; links 8.9 ms at 2, 8.8 at 3 and at 4, and
// on 32x32x64 0.097 ms at 2, 0.115 at 3, 0.086 at 4.)
#ifndef GLASMA_FP64_MIN_BLOCKS
#define GLASMA_FP64_MIN_BLOCKS 2
#endif
#ifndef GLASMA_FP32_MIN_BLOCKS
#define GLASMA_FP32_MIN_BLOCKS 5
#endif
#ifndef GLASMA_FP32_LINKS_MIN_BLOCKS
#define GLASMA_FP32_LINKS_MIN_BLOCKS 8
#endif
#ifndef GLASMA_FP32_FUSED_MIN_BLOCKS
#define GLASMA_FP32_FUSED_MIN_BLOCKS 4
#endif
#ifndef GLASMA_FP32_PLAQ_MIN_BLOCKS
#define GLASMA_FP32_PLAQ_MIN_BLOCKS 4
#endif
#ifndef GLASMA_DDF_PLAQ_MIN_BLOCKS
#define GLASMA_DDF_PLAQ_MIN_BLOCKS 3
#endif
#ifndef GLASMA_FX_LINKS_MIN_BLOCKS
#define GLASMA_FX_LINKS_MIN_BLOCKS 2
#endif
#ifndef GLASMA_FX_PLAQ_MIN_BLOCKS
#define GLASMA_FX_PLAQ_MIN_BLOCKS 3
#endif
template <typename T>
struct Occupancy;
template <>
struct Occupancy<double> {
  static constexpr int kMinBlocks = GLASMA_FP64_MIN_BLOCKS;       // electric-field kernel
  static constexpr int kLinksMinBlocks = GLASMA_FX_LINKS_MIN_BLOCKS;  // link/J kernel
  static constexpr int kFusedMinBlocks = GLASMA_FP64_MIN_BLOCKS;  // one-pass step kernel
  static constexpr int kPlaqMinBlocks = GLASMA_FX_PLAQ_MIN_BLOCKS;  // plaquette-method force kernel
};
template <>
struct Occupancy<float> {
  static constexpr int kMinBlocks = GLASMA_FP32_MIN_BLOCKS;
  static constexpr int kLinksMinBlocks = GLASMA_FP32_LINKS_MIN_BLOCKS;
  static constexpr int kFusedMinBlocks = GLASMA_FP32_FUSED_MIN_BLOCKS;
  static constexpr int kPlaqMinBlocks = GLASMA_FP32_PLAQ_MIN_BLOCKS;
};

template <typename I>
__device__ __forceinline__ I nb(const Geometry& g, int x, int y, int z, int dx, int dy, int dz) {
  int xx = x + dx, yy = y + dy;
  xx = xx < 0 ? xx + g.nx : (xx >= g.nx ? xx - g.nx : xx);
  yy = yy < 0 ? yy + g.ny : (yy >= g.ny ? yy - g.ny : yy);
  return (I)xx + (I)g.nx * ((I)yy + (I)g.ny * (I)(z + dz + 1));
}

template <typename I>
__device__ __forceinline__ void decode(const Geometry& g, I idx, int& x, int& y, int& z) {
  const I r = idx / (I)g.nx;
  x = (int)(idx - r * (I)g.nx);
  z = (int)(r / (I)g.ny);
  y = (int)(r - (I)z * (I)g.ny);
}

// v[mu] for a runtime mu without indexing the kernel-parameter array (which would copy it to the stack)
template <typename T>
__device__ __forceinline__ T pick3(const T (&v)[3], int mu) {
  return mu == 0 ? v[0] : (mu == 1 ? v[1] : v[2]);
}

// acc += c (a - b), componentwise: the update form of UpdateJStat and UpdateJ.  Every path (K1, K2,
// the fused step) uses this one expression, so they round identically.
template <typename T>
__device__ __forceinline__ void axpy_diff(Alg<T>& acc, T c, const Alg<T>& a, const Alg<T>& b) {
#pragma unroll
  for (int k = 0; k < 8; k++) acc.a[k] += c * (a.a[k] - b.a[k]);
}

// FP64 staple sharing: for mu < nu the first product of link mu's upper staple in plane nu,
// A = U_nu(x+mu) U_mu^d(x+nu), is the dagger of the first product of link nu's upper staple in plane
// mu, so it is formed once and parked in the thread's own shared-memory slot until link nu needs it
// (3 of the 27 staple matmuls saved; two slots suffice since the links are processed in order).
// On for FP32 too (measured 5 % faster K1 on GB300; GLASMA_FP32_STAPLE_SHARE=0 turns it off there).  Slot k, element e of thread t: sh[(k*9+e)*kThreads+t].
#ifndef GLASMA_FP32_STAPLE_SHARE
#define GLASMA_FP32_STAPLE_SHARE 1
#endif
template <typename T>
struct StapleShare {
  static constexpr int kSlots = (sizeof(T) == 8 || GLASMA_FP32_STAPLE_SHARE) ? 2 : 0;
};
enum StapleMode { kStapleCompute = 0, kStapleStore = 1, kStapleReuse = 2 };

// Staples of link mu at x in the (mu,nu) plane, weighted by c, added to acc.  R: rows of each link
// stored (3 full, 2 for 12-real links, see load_link_r).
template <typename T, typename I, int R = 3>
__device__ __forceinline__ void add_staples(const cx<T>* __restrict__ U, I S, int mu, int nu, I s, I s_pmu, I s_pnu,
                                            I s_pmu_mnu, I s_mnu, T c, Mat<T>& acc, cx<T>* sh = nullptr,
                                            int mode = kStapleCompute, int slot = 0) {
  Mat<T> a, b, t;
  if (sh && mode == kStapleReuse) {
    const cx<T>* q = sh + (slot * 9) * kThreads + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const cx<T> v = q[(j + 3 * i) * kThreads];
        t.e[i + 3 * j] = mk<T>(v.re, -v.im);
      }
  } else {
    load_link_r<R>(U, S, nu, s_pmu, a);
    load_link_r<R>(U, S, mu, s_pnu, b);
    mul_nd(a, b, t);
    if (sh && mode == kStapleStore) {
      cx<T>* q = sh + (slot * 9) * kThreads + threadIdx.x;
#pragma unroll
      for (int k = 0; k < 9; k++) q[k * kThreads] = t.e[k];
    }
  }
  load_link_r<R>(U, S, nu, s, a);
  add_mul_nd(t, a, c, acc);
  load_link_r<R>(U, S, nu, s_pmu_mnu, a);
  load_link_r<R>(U, S, mu, s_mnu, b);
  mul_dd(a, b, t);
  load_link_r<R>(U, S, nu, s_mnu, a);
  add_mul_nn(t, a, c, acc);
}

template <typename T>
struct EParams {
  T gc[3];    // gamma * cE[mu],   gamma = -2 dt a^3, cE = 1/a_mu^2
  T cnu[3];   // cE[nu]
  T jz;       // -(dt/a_z)/sqrt(2)
  T cj;       // dt/a_z
  int do_e, do_jstat;
  int dry;    // compute, store nothing (autotuner timing runs)
};

// The electric-field and JStat update of one site (K1's per-site body).
template <typename T, typename I, int R = 3>
__device__ __forceinline__ void efield_site(const Geometry& g, const FieldPtrs<T>& f, const EParams<T>& p, int x, int y,
                                            int z, cx<T>* sh = nullptr) {
  const I S = (I)g.S, plane = (I)g.plane;
  const I s = (I)x + (I)g.nx * ((I)y + (I)g.ny * (I)(z + 1));
  const bool lo = (z == 0), hi = (z == g.nz - 1);
  const I sg = lo ? s - plane : (hi ? s + plane : (I)-1);
  if (p.do_e) {
    const I sxp = nb<I>(g, x, y, z, 1, 0, 0), sxm = nb<I>(g, x, y, z, -1, 0, 0);
    const I syp = nb<I>(g, x, y, z, 0, 1, 0), sym = nb<I>(g, x, y, z, 0, -1, 0);
    const I szp = s + plane, szm = s - plane;
#pragma unroll 1
    for (int mu = 0; mu < 3; mu++) {
      Mat<T> acc;
      set_zero(acc);
      if (mu == 0) {
        add_staples<T, I, R>(f.U, S, 0, 1, s, sxp, syp, nb<I>(g, x, y, z, 1, -1, 0), sym, p.cnu[1], acc, sh, kStapleStore, 0);
        add_staples<T, I, R>(f.U, S, 0, 2, s, sxp, szp, nb<I>(g, x, y, z, 1, 0, -1), szm, p.cnu[2], acc, sh, kStapleStore, 1);
      } else if (mu == 1) {
        add_staples<T, I, R>(f.U, S, 1, 0, s, syp, sxp, nb<I>(g, x, y, z, -1, 1, 0), sxm, p.cnu[0], acc, sh, kStapleReuse, 0);
        add_staples<T, I, R>(f.U, S, 1, 2, s, syp, szp, nb<I>(g, x, y, z, 0, 1, -1), szm, p.cnu[2], acc, sh, kStapleStore, 0);
      } else {
        add_staples<T, I, R>(f.U, S, 2, 0, s, szp, sxp, nb<I>(g, x, y, z, -1, 0, 1), sxm, p.cnu[0], acc, sh, kStapleReuse, 1);
        add_staples<T, I, R>(f.U, S, 2, 1, s, szp, syp, nb<I>(g, x, y, z, 0, -1, 1), sym, p.cnu[1], acc, sh, kStapleReuse, 0);
      }
      Mat<T> u, P;
      load_link_r<R>(f.U, S, mu, s, u);
      mul_nn_traceless(u, acc, P);
      Alg<T> force, e;
      retr_itg(P, pick3(p.gc, mu), force);
      load_alg(f.E, S, mu * 8, s, e);
#pragma unroll
      for (int a = 0; a < 8; a++) e.a[a] += force.a[a];
      if (mu == 2) {
        Alg<T> jp, jm;
        load_alg(f.Jp, S, 0, s, jp);
        load_alg(f.Jm, S, 0, s, jm);
#pragma unroll
        for (int a = 0; a < 8; a++) e.a[a] += p.jz * (jp.a[a] - jm.a[a]);
      }
      if (!p.dry) {
        store_alg(f.E, S, mu * 8, s, e);
        if (sg >= 0) store_alg(f.E, S, mu * 8, sg, e);
      }
    }
  }
  if (p.do_jstat) {
    const I szm = s - plane;
    Mat<T> uzm;
    load_link_r<R>(f.U, S, 2, szm, uzm);
    Alg<T> down, downm, jc, st;
    load_alg(f.Jp, S, 0, szm, jc);
    load_alg(f.Jm, S, 0, szm, st);
    rotate_currents<T, false>(uzm, jc, st, down, downm);
    load_alg(f.Jp, S, 0, s, jc);
    load_alg(f.JpStat, S, 0, s, st);
    axpy_diff(st, -p.cj, jc, down);
    if (!p.dry) {
      store_alg(f.JpStat, S, 0, s, st);
      if (sg >= 0) store_alg(f.JpStat, S, 0, sg, st);
    }
    down = downm;
    load_alg(f.Jm, S, 0, s, jc);
    load_alg(f.JmStat, S, 0, s, st);
    axpy_diff(st, p.cj, jc, down);
    if (!p.dry) {
      store_alg(f.JmStat, S, 0, s, st);
      if (sg >= 0) store_alg(f.JmStat, S, 0, sg, st);
    }
  }
}

// ---- the plaquette method --------------------------------------------------------------------------
// The force of UpdateElectricFields is a sum over plaquettes: the plaquette P = a b c^d d^d at y in the
// plane (p, q), p < q (a = U_p(y), b = U_q(y+p), c = U_p(y+q), d = U_q(y)), with al = ReTr(i t P),
// enters four links, as the upper or lower staple of each (c_mu = cE[mu], gc_mu = gamma c_mu):
//   link p at y     +gc_p c_q al                      (U_p(y) S_{+q} = P)
//   link q at y     -gc_q c_p al                      (U_q(y) S_{+p} = P^d)
//   link p at y+q   -gc_p c_q InvAdj(d, al)           (U_p(y+q) S_{-q} = d^d P^d d)
//   link q at y+p   +gc_q c_p InvAdj(a, al)           (U_q(y+p) S_{-p} = a^d P a)
// using ReTr(i t X^d) = -ReTr(i t X) and ReTr(i t^a V^d X V) = InvAdj(V, ReTr(i t X))_a, the SU(3)
// InverseAdjointMultiplication.  The same terms as the staple form (K1), regrouped: three plaquettes
// (three products each) and six adjoint rotations per site instead of twelve staples (two products
// each, three shared) and three final products: ~18 instead of ~24 matrix products per site.
// K1' (plaquette_site_direct, or plaquette_site_fx in FP64) runs one thread per plaquette owner y, slices -1 .. Nz-1
// (the ghost slice owns the plaquettes whose lower-staple terms reach slice 0): it adds the first two terms and the current
// source to E at y and stores the rotated vectors of the last two, without their weights, in a contribution
// buffer at y.  K2' (links_site with kGather) adds the two each link receives, from y = x-q and x-p, times
// their weights (LParams wa, wb: an fma where a weighted contribution would take an add) to E before it
// exponentiates it.  Contribution slots C[(slot*8 + a)*S + y]:
enum ContribSlot {
  kC01p = 0,  // plane (0,1), to link 1 at y+x
  kC01q = 1,  // plane (0,1), to link 0 at y+y
  kC02p = 2,  // plane (0,2), to link 2 at y+x
  kC02q = 3,  // plane (0,2), to link 0 at y+z
  kC12p = 4,  // plane (1,2), to link 2 at y+y
  kC12q = 5,  // plane (1,2), to link 1 at y+z
  kCSlots = 6
};

template <typename T>
__device__ __forceinline__ void scale_alg(T w, Alg<T>& v) {
#pragma unroll
  for (int k = 0; k < 8; k++) v.a[k] *= w;
}

// al = ReTr(i t^a a b c^d d^d)
template <typename T>
__device__ __forceinline__ void plaquette_alg(const Mat<T>& a, const Mat<T>& b, const Mat<T>& c, const Mat<T>& d,
                                              Alg<T>& al) {
  Mat<T> ab, dc, P;
  mul_nn(a, b, ab);
  mul_nn(d, c, dc);
  mul_nd_traceless(ab, dc, P);
  retr_itg(P, T(1), al);
}

// K1' per owner site: idx = owner site s (slice -1 starts at s = 0); covers (Nz+1) slices.  TC is the
// arithmetic type: T itself, or ddf for FP64 fields (double-float arithmetic on the FP32 pipe, the
// fields converted on load and store).
template <typename T, typename I, int R, typename TC = T>
__device__ __forceinline__ void plaquette_site_direct(const Geometry& g, const FieldPtrs<T>& f, T* __restrict__ C,
                                                      const EParams<T>& p, I idx) {
  const I S = (I)g.S, plane = (I)g.plane;
  const I s = idx;
  const int zz = (int)(idx / plane);
  const int z = zz - 1;
  const int r = (int)(idx - (I)zz * plane);
  const int y = r / g.nx, x = r - y * g.nx;
  const bool interior = z >= 0;
  const bool below_top = z < g.nz - 1;  // y+z is an interior site
  const I sxp = nb<I>(g, x, y, z, 1, 0, 0), syp = nb<I>(g, x, y, z, 0, 1, 0), szp = s + plane;
  // wp = gc_p c_q, wq = gc_q c_p (formed in the storage type, then converted)
  const TC w01p = to_compute<TC>(p.gc[0] * p.cnu[1]), w01q = to_compute<TC>(p.gc[1] * p.cnu[0]);
  const TC w02p = to_compute<TC>(p.gc[0] * p.cnu[2]), w02q = to_compute<TC>(p.gc[2] * p.cnu[0]);
  const TC w12p = to_compute<TC>(p.gc[1] * p.cnu[2]), w12q = to_compute<TC>(p.gc[2] * p.cnu[1]);
  Alg<TC> F0, F1, F2, al, out;
  Mat<TC> u0, u1, u2, b, c;
  load_link_c<R>(f.U, S, 0, s, u0);
  load_link_c<R>(f.U, S, 1, s, u1);
  load_link_c<R>(f.U, S, 2, s, u2);
  if constexpr (kPairRotations<TC>) {
    // the three plaquettes first, then the six rotations in pairs by the same link:
    // u1 (al01 -> link 0 at y+y, al12 -> link 2 at y+y), u0 (al01 -> link 1 at y+x, al02 -> link 2 at
    // y+x), u2 (al02 -> link 0 at y+z, al12 -> link 1 at y+z)
    Alg<TC> al01, al12, out2;
    if (interior) {
      // plane (0,1): a = U_0(y), b = U_1(y+x), c = U_0(y+y), d = U_1(y)
      load_link_c<R>(f.U, S, 1, sxp, b);
      load_link_c<R>(f.U, S, 0, syp, c);
      plaquette_alg(u0, b, c, u1, al01);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        F0.a[k] = w01p * al01.a[k];
        F1.a[k] = -w01q * al01.a[k];
      }
    }
    // plane (0,2): a = U_0(y), b = U_2(y+x), c = U_0(y+z), d = U_2(y)
    load_link_c<R>(f.U, S, 2, sxp, b);
    load_link_c<R>(f.U, S, 0, szp, c);
    plaquette_alg(u0, b, c, u2, al);
    // plane (1,2): a = U_1(y), b = U_2(y+y), c = U_1(y+z), d = U_2(y)
    load_link_c<R>(f.U, S, 2, syp, b);
    load_link_c<R>(f.U, S, 1, szp, c);
    plaquette_alg(u1, b, c, u2, al12);
    if (below_top) {
      inv_adj_mul2(u2, al, al12, out, out2);
      if (!p.dry) {
        store_alg_c(C, S, kC02q * 8, s, out);
        store_alg_c(C, S, kC12q * 8, s, out2);
      }
    }
    if (!interior) return;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      F0.a[k] += w02p * al.a[k];
      F2.a[k] = -w02q * al.a[k];
      F1.a[k] += w12p * al12.a[k];
      F2.a[k] -= w12q * al12.a[k];
    }
    inv_adj_mul2(u1, al01, al12, out, out2);
    if (!p.dry) {
      store_alg_c(C, S, kC01q * 8, s, out);
      store_alg_c(C, S, kC12p * 8, s, out2);
    }
    inv_adj_mul2(u0, al01, al, out, out2);
    if (!p.dry) {
      store_alg_c(C, S, kC01p * 8, s, out);
      store_alg_c(C, S, kC02p * 8, s, out2);
    }
  } else {
    if (interior) {
      // plane (0,1): a = U_0(y), b = U_1(y+x), c = U_0(y+y), d = U_1(y)
      load_link_c<R>(f.U, S, 1, sxp, b);
      load_link_c<R>(f.U, S, 0, syp, c);
      plaquette_alg(u0, b, c, u1, al);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        F0.a[k] = w01p * al.a[k];
        F1.a[k] = -w01q * al.a[k];
      }
      inv_adj_mul(u1, al, out);  // to link 0 at y+y
      if (!p.dry) store_alg_c(C, S, kC01q * 8, s, out);
      inv_adj_mul(u0, al, out);  // to link 1 at y+x
      if (!p.dry) store_alg_c(C, S, kC01p * 8, s, out);
    }
    // plane (0,2): a = U_0(y), b = U_2(y+x), c = U_0(y+z), d = U_2(y)
    load_link_c<R>(f.U, S, 2, sxp, b);
    load_link_c<R>(f.U, S, 0, szp, c);
    plaquette_alg(u0, b, c, u2, al);
    if (below_top) {
      inv_adj_mul(u2, al, out);  // to link 0 at y+z
      if (!p.dry) store_alg_c(C, S, kC02q * 8, s, out);
    }
    if (interior) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        F0.a[k] += w02p * al.a[k];
        F2.a[k] = -w02q * al.a[k];
      }
      inv_adj_mul(u0, al, out);  // to link 2 at y+x
      if (!p.dry) store_alg_c(C, S, kC02p * 8, s, out);
    }
    // plane (1,2): a = U_1(y), b = U_2(y+y), c = U_1(y+z), d = U_2(y)
    load_link_c<R>(f.U, S, 2, syp, b);
    load_link_c<R>(f.U, S, 1, szp, c);
    plaquette_alg(u1, b, c, u2, al);
    if (below_top) {
      inv_adj_mul(u2, al, out);  // to link 1 at y+z
      if (!p.dry) store_alg_c(C, S, kC12q * 8, s, out);
    }
    if (!interior) return;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      F1.a[k] += w12p * al.a[k];
      F2.a[k] -= w12q * al.a[k];
    }
    inv_adj_mul(u1, al, out);  // to link 2 at y+y
    if (!p.dry) store_alg_c(C, S, kC12p * 8, s, out);
  }
  // E += the forces of the plaquettes owned here (+ the current source on E_z); K2' adds the rest
  Alg<TC> e;
  load_alg_c(f.E, S, 0, s, e);
#pragma unroll
  for (int k = 0; k < 8; k++) e.a[k] += F0.a[k];
  if (!p.dry) store_alg_c(f.E, S, 0, s, e);
  load_alg_c(f.E, S, 8, s, e);
#pragma unroll
  for (int k = 0; k < 8; k++) e.a[k] += F1.a[k];
  if (!p.dry) store_alg_c(f.E, S, 8, s, e);
  {
    Alg<TC> jp, jm;
    const TC jz = to_compute<TC>(p.jz);
    load_alg_c(f.E, S, 16, s, e);
    load_alg_c(f.Jp, S, 0, s, jp);
    load_alg_c(f.Jm, S, 0, s, jm);
#pragma unroll
    for (int k = 0; k < 8; k++) e.a[k] += F2.a[k] + jz * (jp.a[k] - jm.a[k]);
    if (!p.dry) store_alg_c(f.E, S, 16, s, e);
  }
  // UpdateJStat, as K1
  const bool lo = (z == 0), hi = (z == g.nz - 1);
  const I sg = lo ? s - plane : (hi ? s + plane : (I)-1);
  const I szm = s - plane;
  const TC cj = to_compute<TC>(p.cj);
  Mat<TC> uzm;
  load_link_c<R>(f.U, S, 2, szm, uzm);
  Alg<TC> down, downm, jc, st;
  load_alg_c(f.Jp, S, 0, szm, jc);
  if constexpr (kPairRotations<TC>) {
    load_alg_c(f.Jm, S, 0, szm, st);
    rotate_currents<TC, false>(uzm, jc, st, down, downm);
  } else {
    inv_adj_mul(uzm, jc, down);
  }
  load_alg_c(f.Jp, S, 0, s, jc);
  load_alg_c(f.JpStat, S, 0, s, st);
  axpy_diff(st, -cj, jc, down);
  if (!p.dry) {
    store_alg_c(f.JpStat, S, 0, s, st);
    if (sg >= 0) store_alg_c(f.JpStat, S, 0, sg, st);
  }
  if constexpr (kPairRotations<TC>) {
    down = downm;
  } else {
    load_alg_c(f.Jm, S, 0, szm, jc);
    inv_adj_mul(uzm, jc, down);
  }
  load_alg_c(f.Jm, S, 0, s, jc);
  load_alg_c(f.JmStat, S, 0, s, st);
  axpy_diff(st, cj, jc, down);
  if (!p.dry) {
    store_alg_c(f.JmStat, S, 0, s, st);
    if (sg >= 0) store_alg_c(f.JmStat, S, 0, sg, st);
  }
}

// plaquette_site_direct for FP64 fields with the products on the integer pipe (fx.cuh).  Bound by FP64, the direct form
// runs ~2000 FP64 operations per site; here they are ~5,000 mad.wide and ~15,000 other integer operations, with ~300
// FP64 ones beside them (the sums into E, conversions): 128x128x512 30.7 ms in FP64, 10.9 here.  One copy of the plaquette
// and of the rotation in the code, so that it stays inside the instruction cache; the three anti-Hermitian parts wait in
// shared memory for their rotations.
// kRoles = 1: a thread does its site's three plaquettes and four rotation pairs in turn.  kRoles = 4: a block of four
// warps does 32 sites, warp r plaquette r, rotation r and the sum into E_r (warp 3 the currents' rotation and JStat):
// a third of the serial chain and four times the blocks, for lattices that do not fill the GPU (launch_plaquette_rows).
// The arithmetic is the same either way.  Sites that the fixed-point format does not hold go through the FP64 form.
template <typename I>
static __device__ __noinline__ void plaquette_site_fp64(const Geometry& g, const FieldPtrs<double>& f, double* C,
                                                 const EParams<double>& p, I idx) {
  plaquette_site_direct<double, I, 3>(g, f, C, p, idx);
}

template <int kRoles>
constexpr int kFxSites = kThreads / kRoles;  // sites per block
template <int kRoles>
constexpr int kFxShared = (3 * 18 + 3 + (kRoles > 1 ? kRoles : 0)) * kFxSites<kRoles>;  // ints of shared memory per block

template <typename I, int kRoles>
__device__ __forceinline__ void plaquette_site_fx(const Geometry& g, const FieldPtrs<double>& f, double* __restrict__ C,
                                                  const EParams<double>& p, I idx, bool active, int role,
                                                  int* __restrict__ sh) {
  using fx::ll;
  constexpr int kSites = kFxSites<kRoles>;
  const I S = (I)g.S, plane = (I)g.plane;
  const I s = idx;
  const int zz = (int)(idx / plane);
  const int z = zz - 1;
  const int r = (int)(idx - (I)zz * plane);
  const int y = r / g.nx, x = r - y * g.nx;
  const bool interior = z >= 0;
  const bool below_top = z < g.nz - 1;
  const int site = kRoles == 1 ? threadIdx.x : threadIdx.x % kSites;
  ll* const slot = reinterpret_cast<ll*>(sh) + site;  // number w of plane n: slot[(n * 9 + w) * kSites]
  int* const slot_e = sh + 3 * 18 * kSites + site;
  int* const flag = slot_e + 3 * kSites;  // kRoles > 1: role r's guard
  auto put = [&](int n, const fx::Anti& a) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      slot[(n * 9 + k) * kSites] = a.y[k];
      slot[(n * 9 + 3 + k) * kSites] = a.x[k];
      slot[(n * 9 + 6 + k) * kSites] = a.d[k];
    }
    slot_e[n * kSites] = a.e;
  };
  auto get = [&](int n, fx::Anti& a) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      a.y[k] = slot[(n * 9 + k) * kSites];
      a.x[k] = slot[(n * 9 + 3 + k) * kSites];
      a.d[k] = slot[(n * 9 + 6 + k) * kSites];
    }
    a.e = slot_e[n * kSites];
  };
  fx::Guard guard = fx::guard_init();
  // planes 0: (0,1), 1: (0,2), 2: (1,2); the ghost slice -1 owns only those with z
  auto plaquette = [&](int n) {
    const int mp = n == 2 ? 1 : 0, mq = n == 0 ? 1 : 2;
    const I sp = n == 2 ? nb<I>(g, x, y, z, 0, 1, 0) : nb<I>(g, x, y, z, 1, 0, 0);
    const I sq = n == 0 ? nb<I>(g, x, y, z, 0, 1, 0) : s + plane;
    fx::M a, b, w, v;
    int ea, eb, ew, ev;
    fx::link_near(f.U, S, mp, s, a, ea, guard);
    fx::link_near(f.U, S, mq, sp, b, eb, guard);
    fx::near_product(a, ea, b, eb, w, ew, guard);
    fx::link_near(f.U, S, mq, s, a, ea, guard);
    fx::link_near(f.U, S, mp, sq, b, eb, guard);
    fx::near_product(a, ea, b, eb, v, ev, guard);
    fx::Anti al;
    fx::plaquette_parts(w, ew, v, ev, al);
    put(n, al);
  };
  // rotations: 0 by u2 (al02, al12), 1 by u1 (al01, al12), 2 by u0 (al01, al02), 3 the currents below by U_2(y-z)
  Alg<double> down, downm;
  auto rotation = [&](int n) {
    fx::M v, m;
    int e;
    ll o1[8], o2[8];
    fx::link_plain(f.U, S, n == 3 ? 2 : 2 - n, n == 3 ? s - plane : s, v, guard);
    if (n < 3) {
      fx::Anti a1, a2;
      get(n == 0 ? 1 : 0, a1);
      get(n == 2 ? 1 : 2, a2);
      fx::herm_pair(a1, a2, m, e);
    } else {
      Alg<double> jp, jm;
      load_alg(f.Jp, S, 0, s - plane, jp);
      load_alg(f.Jm, S, 0, s - plane, jm);
      fx::herm_pair(jp, jm, m, e, guard);
    }
    fx::rotate_pair<true>(v, m, o1, o2, guard);
    if (n < 3) {
      const int k1 = n == 0 ? kC02q : (n == 1 ? kC01q : kC01p), k2 = n == 0 ? kC12q : (n == 1 ? kC12p : kC02p);
      Alg<double> out, out2;
      fx::to_alg<true>(o1, e - fx::kScale - 2, -1.0, out);
      fx::to_alg<true>(o2, e - fx::kScale - 2, -1.0, out2);
      if (!p.dry) {
        store_alg(C, S, k1 * 8, s, out);
        store_alg(C, S, k2 * 8, s, out2);
      }
    } else {
      fx::to_alg<true>(o1, e - fx::kScale - 1, 1.0, down);
      fx::to_alg<true>(o2, e - fx::kScale - 1, 1.0, downm);
    }
  };
  // -2 al of plane n as doubles; with one role they then wait in the place of the fixed-point form, for two links
  auto convert = [&](int n, Alg<double>& v) {
    fx::Anti a;
    get(n, a);
#pragma unroll
    for (int k = 0; k < 8; k++) v.a[k] = fx::from_fixed_fp64(fx::component(a, k), a.e - fx::kScale);
    v.a[7] *= Consts<double>::inv_sqrt3();
  };
  auto alg = [&](int n, Alg<double>& v) {
    if constexpr (kRoles == 1) {
#pragma unroll
      for (int k = 0; k < 8; k++) v.a[k] = __longlong_as_double(slot[(n * 9 + k) * kSites]);
    } else {
      convert(n, v);
    }
  };
  // E_mu += the forces of the plaquettes owned here (+ the current source on E_z)
  auto efield = [&](int mu) {
    // link 0: +w01p al01 + w02p al02; link 1: -w01q al01 + w12p al12; link 2: -w02q al02 - w12q al12
    // (w_pq p = gc_p c_q, q = gc_q c_p)
    const int n1 = mu == 2 ? 1 : 0, n2 = mu == 0 ? 1 : 2;
    const double c1 = -0.5 * (mu == 0 ? p.gc[0] * p.cnu[1] : (mu == 1 ? -(p.gc[1] * p.cnu[0]) : -(p.gc[2] * p.cnu[0])));
    const double c2 = -0.5 * (mu == 0 ? p.gc[0] * p.cnu[2] : (mu == 1 ? p.gc[1] * p.cnu[2] : -(p.gc[2] * p.cnu[1])));
    Alg<double> e, F, v1, v2;
    load_alg(f.E, S, mu * 8, s, e);
    alg(n1, v1);
    alg(n2, v2);
#pragma unroll
    for (int k = 0; k < 8; k++) F.a[k] = fma(v2.a[k], c2, v1.a[k] * c1);
    if (mu == 2) {
      Alg<double> jp, jm;
      load_alg(f.Jp, S, 0, s, jp);
      load_alg(f.Jm, S, 0, s, jm);
#pragma unroll
      for (int k = 0; k < 8; k++) F.a[k] += p.jz * (jp.a[k] - jm.a[k]);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) e.a[k] += F.a[k];
    if (!p.dry) store_alg(f.E, S, mu * 8, s, e);
  };
  auto jstat = [&]() {  // UpdateJStat, as K1
    const bool lo = (z == 0), hi = (z == g.nz - 1);
    const I sg = lo ? s - plane : (hi ? s + plane : (I)-1);
    Alg<double> jc, st;
    load_alg(f.Jp, S, 0, s, jc);
    load_alg(f.JpStat, S, 0, s, st);
    axpy_diff(st, -p.cj, jc, down);
    if (!p.dry) {
      store_alg(f.JpStat, S, 0, s, st);
      if (sg >= 0) store_alg(f.JpStat, S, 0, sg, st);
    }
    load_alg(f.Jm, S, 0, s, jc);
    load_alg(f.JmStat, S, 0, s, st);
    axpy_diff(st, p.cj, jc, downm);
    if (!p.dry) {
      store_alg(f.JmStat, S, 0, s, st);
      if (sg >= 0) store_alg(f.JmStat, S, 0, sg, st);
    }
  };
  // Neither E nor JStat is written before every guard of the site is known.
  if constexpr (kRoles == 1) {
    if (!active) return;
#pragma unroll 1
    for (int n = interior ? 0 : 1; n < 3; n++) plaquette(n);
#pragma unroll 1
    for (int n = below_top ? 0 : 1; n < (interior ? 4 : 1); n++) rotation(n);
    if (fx::tripped(guard)) {
      plaquette_site_fp64<I>(g, f, C, p, idx);
      return;
    }
    if (!interior) return;
#pragma unroll 1
    for (int n = 0; n < 3; n++) {
      Alg<double> v;
      convert(n, v);
#pragma unroll
      for (int k = 0; k < 8; k++) slot[(n * 9 + k) * kSites] = __double_as_longlong(v.a[k]);
    }
#pragma unroll 1
    for (int mu = 0; mu < 3; mu++) efield(mu);
    jstat();
  } else {
    if (active && role < 3 && (interior || role > 0)) plaquette(role);
    __syncthreads();
    // role 3's rotation reads no plaquette; it waits here only so that the rotation is in the code once
    if (active && (role == 0 ? below_top : interior)) rotation(role);
    flag[role * kSites] = active && fx::tripped(guard);
    __syncthreads();
    if (!active) return;
    if (flag[0] | flag[kSites] | flag[2 * kSites] | flag[3 * kSites]) {
      if (role == 0) plaquette_site_fp64<I>(g, f, C, p, idx);
      return;
    }
    if (!interior) return;
    if (role < 3)
      efield(role);
    else
      jstat();
  }
}

// Ints of shared memory the force kernel of type T, TC needs per block.
template <typename T, typename TC, int kRoles>
constexpr int kPlaqShared = (std::is_same<T, double>::value && std::is_same<TC, double>::value) ? kFxShared<kRoles> : 2;

// One block of the force kernel over n owner sites, block b.
template <typename T, typename I, int R, typename TC, int kRoles = 1>
__device__ __forceinline__ void plaquette_block(const Geometry& g, const FieldPtrs<T>& f, T* __restrict__ C,
                                                const EParams<T>& p, long long b, long long n, int* sh) {
  if constexpr (std::is_same<T, double>::value && std::is_same<TC, double>::value) {
    constexpr int kSites = kFxSites<kRoles>;
    const long long idx = b * kSites + threadIdx.x % kSites;
    // the roles move on by one from block to block, so that no scheduler gets the lighter one every time
    const int role = kRoles == 1 ? 0 : (int)((threadIdx.x / kSites + b) % kRoles);
    plaquette_site_fx<I, kRoles>(g, f, C, p, (I)(idx < n ? idx : 0), idx < n, role, sh);
  } else {
    const long long idx = b * kThreads + threadIdx.x;
    if (idx < n) plaquette_site_direct<T, I, R, TC>(g, f, C, p, (I)idx);
  }
}

// Blocks per SM of the force kernel: by storage type, and for FP64 fields computed in double-float.
template <typename T, typename TC>
struct PlaqOccupancy {
  static constexpr int kMinBlocks = Occupancy<T>::kPlaqMinBlocks;
};
template <>
struct PlaqOccupancy<double, ddf> {
  static constexpr int kMinBlocks = GLASMA_DDF_PLAQ_MIN_BLOCKS;
};

// Thread-to-site map of K1: a block of kThreads threads covers a tile of tile_x x (kThreads/tile_x)
// sites of one z slice, so most y-neighbours a block reads are its own sites (L1 hits).
struct TileMap {
  int tile_x, tile_y, ntx, nty;
  __host__ __device__ static TileMap make(int nx, int ny, int tile_x, int threads) {
    TileMap t;
    t.tile_x = tile_x;
    t.tile_y = threads / tile_x;
    t.ntx = (nx + t.tile_x - 1) / t.tile_x;
    t.nty = (ny + t.tile_y - 1) / t.tile_y;
    return t;
  }
  __host__ __device__ long long tiles(int nz) const { return (long long)ntx * nty * nz; }
  // tile index -> site of thread `t` (false when the thread falls outside the lattice)
  __device__ bool site(long long tile, int t, int nx, int ny, int& x, int& y, int& z) const {
    const long long per_z = (long long)ntx * nty;
    z = (int)(tile / per_z);
    const int r = (int)(tile - (long long)z * per_z);
    const int by = r / ntx, bx = r - by * ntx;
    x = bx * tile_x + t % tile_x;
    y = by * tile_y + t / tile_x;
    return x < nx && y < ny;
  }
};

template <typename T>
struct LParams {
  T cU[3];  // -(h) a_mu^2 / a^3 for the half step h
  T cj;     // dt/a_z
  T wa[3], wb[3];  // plaquette method: weights of the two contributions link mu gathers
  int save_uold, do_j, do_second;
};

// Weights of the contributions: gc_p c_q and gc_q c_p with gc_mu = gamma c_mu, gamma = -2 dt a^3, c_mu = 1 / a_mu^2,
// formed in the fields' precision.  Link 0 gathers (0,1) from x-y and (0,2) from x-z, link 1 (0,1) from x-x and (1,2)
// from x-z, link 2 (0,2) from x-x and (1,2) from x-y.
template <typename T>
inline void set_gather_weights(const Geometry& g, double dt, LParams<T>& p) {
  const double gamma = -2.0 * dt * (g.a[0] * g.a[1] * g.a[2]);
  T gc[3], c[3];
  for (int mu = 0; mu < 3; mu++) {
    const double ce = 1.0 / (g.a[mu] * g.a[mu]);
    gc[mu] = (T)(gamma * ce);
    c[mu] = (T)ce;
  }
  p.wa[0] = -(gc[0] * c[1]);
  p.wb[0] = -(gc[0] * c[2]);
  p.wa[1] = gc[1] * c[0];
  p.wb[1] = -(gc[1] * c[2]);
  p.wa[2] = gc[2] * c[0];
  p.wb[2] = gc[2] * c[1];
}

// UpdateJ at s with the z link uh of t + dt/2.
template <typename T, typename I>
__device__ __forceinline__ void transport_currents(const FieldPtrs<T>& f, const LParams<T>& p, I S, I s, I szp, I sg,
                                                   const Mat<T>& uh) {
  Alg<T> up, um, st, j;
  load_alg(f.JpStat, S, 0, szp, st);
  if constexpr (kPairCurrents<T>) {
    load_alg(f.JmStat, S, 0, szp, j);
    rotate_currents<T, true>(uh, st, j, up, um);
  } else {
    adj_mul(uh, st, up);
  }
  load_alg(f.JpStat, S, 0, s, st);
  load_alg(f.Jp, S, 0, s, j);
  axpy_diff(j, -p.cj, up, st);
  store_alg(f.Jp, S, 0, s, j);
  if (sg >= 0) store_alg(f.Jp, S, 0, sg, j);
  if constexpr (kPairCurrents<T>) {
    up = um;
  } else {
    load_alg(f.JmStat, S, 0, szp, st);
    adj_mul(uh, st, up);
  }
  load_alg(f.JmStat, S, 0, s, st);
  load_alg(f.Jm, S, 0, s, j);
  axpy_diff(j, p.cj, up, st);
  store_alg(f.Jm, S, 0, s, j);
  if (sg >= 0) store_alg(f.Jm, S, 0, sg, j);
}

// K2's body for link mu of one site: the link to t+dt (two applications of one exp), UOld, J transport (mu = 2).
// kGather (the plaquette method): first E_mu += the two contributions link mu receives from the plaquette owners
// x-nu (see plaquette_site_direct), stored with its ghost copy.
template <typename T, typename I, int R = 3, bool kGather = false>
__device__ __forceinline__ void link_site(const Geometry& g, const FieldPtrs<T>& f, const LParams<T>& p, I idx,
                                           const int mu, const T* __restrict__ C = nullptr) {
  const I S = (I)g.S, plane = (I)g.plane;
  const I s = idx + plane;
  const int z = (int)(idx / plane);
  const bool lo = (z == 0), hi = (z == g.nz - 1);
  const I sg = lo ? s - plane : (hi ? s + plane : (I)-1);
  I sxm = 0, sym = 0;
  if constexpr (kGather) {
    const int r = (int)(idx - (I)z * plane);
    const int y = r / g.nx, x = r - y * g.nx;
    sxm = nb<I>(g, x, y, z, -1, 0, 0);
    sym = nb<I>(g, x, y, z, 0, -1, 0);
  }
  Alg<T> e;
  load_alg(f.E, S, mu * 8, s, e);
  if constexpr (kGather) {
    // link 0: from (0,1) at x-y and (0,2) at x-z; link 1: (0,1) at x-x, (1,2) at x-z;
    // link 2: (0,2) at x-x, (1,2) at x-y
    const I s1 = mu == 0 ? sym : sxm;
    const I s2 = mu == 2 ? sym : s - plane;
    const int c1 = mu == 0 ? kC01q : (mu == 1 ? kC01p : kC02p);
    const int c2 = mu == 0 ? kC02q : (mu == 1 ? kC12q : kC12p);
    Alg<T> a1, a2;
    load_alg(C, S, c1 * 8, s1, a1);
    load_alg(C, S, c2 * 8, s2, a2);
#pragma unroll
    for (int k = 0; k < 8; k++) e.a[k] += fma(pick3(p.wa, mu), a1.a[k], pick3(p.wb, mu) * a2.a[k]);
    store_alg(f.E, S, mu * 8, s, e);
    if (sg >= 0) store_alg(f.E, S, mu * 8, sg, e);
  }
  if constexpr (std::is_same<T, double>::value) {
    // One copy of the product and of the current transport in the code, run once or twice per link: written out
    // (three products, two exponentials) the fixed-point body overflowed the instruction cache (5.6 fetch stalls
    // per issue, 14.3 ms at 128x128x512 where the other form took 10.6; 8.9 now, 21.9 in FP64).
    const bool doubled = p.do_second && !p.save_uold && !(mu == 2 && p.do_j);
    LinkStep<double> X;
    X.set(doubled ? 2.0 * pick3(p.cU, mu) : pick3(p.cU, mu), e);
    Mat<double> u;
    load_link(f.U, S, mu, s, u);
    const int napply = (doubled || !p.do_second) ? 1 : 2;
#pragma unroll 1
    for (int ap = 0; ap < napply; ap++) {
      X.apply(u, u);
      if (ap == 0 && !doubled) {
        if (p.save_uold) {
          store_link(f.UOld, S, mu, s, u);
          if (sg >= 0) store_link(f.UOld, S, mu, sg, u);
        }
        if (mu == 2 && p.do_j) transport_currents<double, I>(f, p, S, s, s + plane, sg, u);
      }
    }
    store_link(f.U, S, mu, s, u);
    if (sg >= 0) store_link(f.U, S, mu, sg, u);
    return;
  }
  LinkStep<T> X;
  Mat<T> u, uh;
  load_link_r<R>(f.U, S, mu, s, u);
  // Without a use for U(t+dt/2) (UOld, the z-link J transport), the two half steps are one:
  // exp(i c t.E)^2 = exp(2i c t.E), one matmul less (equal up to rounding).
  if (p.do_second && !p.save_uold && !(mu == 2 && p.do_j)) {
    X.set(T(2) * pick3(p.cU, mu), e);
    X.apply(u, uh);
    store_link_r<R>(f.U, S, mu, s, uh);
    if (sg >= 0) store_link_r<R>(f.U, S, mu, sg, uh);
    return;
  }
  X.set(pick3(p.cU, mu), e);
  X.apply(u, uh);
  if (p.save_uold) {
    store_link(f.UOld, S, mu, s, uh);
    if (sg >= 0) store_link(f.UOld, S, mu, sg, uh);
  }
  if (mu == 2 && p.do_j) transport_currents<T, I>(f, p, S, s, s + plane, sg, uh);
  if (p.do_second) {
    X.apply(uh, u);
  } else {
    u = uh;
  }
  store_link_r<R>(f.U, S, mu, s, u);
  if (sg >= 0) store_link_r<R>(f.U, S, mu, sg, u);
}

// K2 over the three links of a site in turn.
template <typename T, typename I, int R = 3, bool kGather = false>
__device__ __forceinline__ void links_site(const Geometry& g, const FieldPtrs<T>& f, const LParams<T>& p, I idx,
                                           const T* __restrict__ C = nullptr) {
#pragma unroll 1
  for (int mu = 0; mu < 3; mu++) link_site<T, I, R, kGather>(g, f, p, idx, mu, C);
}

// ---- the whole step in one pass -------------------------------------------------------------------
// fused_site reads the links, currents and static currents of time t from `in` and writes those of
// t+dt to `out` (a second set of buffers; E is updated in place, it is read only at its own site).
// Because nothing it reads is written in the same launch, the sites are independent and the step is
// one launch.  The static currents of t+dt at x+z, which UpdateJ at x needs, are recomputed here from
// the inputs with K1's own expression, so the result is bit-identical to K1 followed by K2.
//   E_mu(x)      += force(U(t)) [+ J term]                          UpdateElectricFields
//   JStat(x)     += -/+ cj (J(x) - U_z^d(x-z) J(x-z) U_z(x-z))      UpdateJStat (also at x+z)
//   Uh            = exp(i cU E_mu(x)) U_mu(x)                        UpdateGaugeLinks(dt/2)
//   J(x)         += -/+ cj (Uh_z J Stat(x+z) Uh_z^d - JStat(x))     UpdateJ
//   U_mu(x; t+dt) = exp(i cU E_mu(x)) Uh                             UpdateGaugeLinks(dt/2)
template <typename T, typename I, int R = 3>
__device__ __forceinline__ void fused_currents(const FieldPtrs<T>& in, const FieldPtrs<T>& out, I S, I plane, I s,
                                               I sg, bool hi, const Mat<T>& uz, const Mat<T>& uhz, T cj, bool dry) {
  const I szm = s - plane, szp = s + plane;
  Alg<T> jc, down, downm, sp, sm;
  {
    Mat<T> w;
    load_link_r<R>(in.U, S, 2, szm, w);
    load_alg(in.Jp, S, 0, szm, jc);
    load_alg(in.Jm, S, 0, szm, sm);
    rotate_currents<T, false>(w, jc, sm, down, downm);
    load_alg(in.Jp, S, 0, s, jc);
    load_alg(in.JpStat, S, 0, s, sp);
    axpy_diff(sp, -cj, jc, down);
    load_alg(in.Jm, S, 0, s, jc);
    load_alg(in.JmStat, S, 0, s, sm);
    axpy_diff(sm, cj, jc, downm);
  }
  if (!dry) {
    store_alg(out.JpStat, S, 0, s, sp);
    store_alg(out.JmStat, S, 0, s, sm);
    if (sg >= 0) {
      store_alg(out.JpStat, S, 0, sg, sp);
      store_alg(out.JmStat, S, 0, sg, sm);
    }
  }
  // static currents of t+dt one slice up (the ghost copy of this site's at the top slice)
  Alg<T> up, um;
  if (hi) {
    up = sp;
    um = sm;
  } else {
    load_alg(in.Jp, S, 0, s, jc);
    load_alg(in.Jm, S, 0, s, um);
    rotate_currents<T, false>(uz, jc, um, down, downm);
    load_alg(in.Jp, S, 0, szp, jc);
    load_alg(in.JpStat, S, 0, szp, up);
    axpy_diff(up, -cj, jc, down);
    load_alg(in.Jm, S, 0, szp, jc);
    load_alg(in.JmStat, S, 0, szp, um);
    axpy_diff(um, cj, jc, downm);
  }
  Alg<T> t, tm, j;
  rotate_currents<T, true>(uhz, up, um, t, tm);
  load_alg(in.Jp, S, 0, s, j);
  axpy_diff(j, -cj, t, sp);
  if (!dry) {
    store_alg(out.Jp, S, 0, s, j);
    if (sg >= 0) store_alg(out.Jp, S, 0, sg, j);
  }
  t = tm;
  load_alg(in.Jm, S, 0, s, j);
  axpy_diff(j, cj, t, sm);
  if (!dry) {
    store_alg(out.Jm, S, 0, s, j);
    if (sg >= 0) store_alg(out.Jm, S, 0, sg, j);
  }
}

template <typename T, typename I, int R = 3>
__device__ __forceinline__ void fused_site(const Geometry& g, const FieldPtrs<T>& in, const FieldPtrs<T>& out,
                                           const EParams<T>& pe, const LParams<T>& pl, int x, int y, int z,
                                           cx<T>* sh = nullptr) {
  const I S = (I)g.S, plane = (I)g.plane;
  const I s = (I)x + (I)g.nx * ((I)y + (I)g.ny * (I)(z + 1));
  const bool lo = (z == 0), hi = (z == g.nz - 1);
  const I sg = lo ? s - plane : (hi ? s + plane : (I)-1);
  const bool dry = pe.dry != 0;
  const I sxp = nb<I>(g, x, y, z, 1, 0, 0), sxm = nb<I>(g, x, y, z, -1, 0, 0);
  const I syp = nb<I>(g, x, y, z, 0, 1, 0), sym = nb<I>(g, x, y, z, 0, -1, 0);
  const I szp = s + plane, szm = s - plane;
#pragma unroll 1
  for (int mu = 0; mu < 3; mu++) {
    Mat<T> acc;
    set_zero(acc);
    if (mu == 0) {
      add_staples<T, I, R>(in.U, S, 0, 1, s, sxp, syp, nb<I>(g, x, y, z, 1, -1, 0), sym, pe.cnu[1], acc, sh, kStapleStore, 0);
      add_staples<T, I, R>(in.U, S, 0, 2, s, sxp, szp, nb<I>(g, x, y, z, 1, 0, -1), szm, pe.cnu[2], acc, sh, kStapleStore, 1);
    } else if (mu == 1) {
      add_staples<T, I, R>(in.U, S, 1, 0, s, syp, sxp, nb<I>(g, x, y, z, -1, 1, 0), sxm, pe.cnu[0], acc, sh, kStapleReuse, 0);
      add_staples<T, I, R>(in.U, S, 1, 2, s, syp, szp, nb<I>(g, x, y, z, 0, 1, -1), szm, pe.cnu[2], acc, sh, kStapleStore, 0);
    } else {
      add_staples<T, I, R>(in.U, S, 2, 0, s, szp, sxp, nb<I>(g, x, y, z, -1, 0, 1), sxm, pe.cnu[0], acc, sh, kStapleReuse, 1);
      add_staples<T, I, R>(in.U, S, 2, 1, s, szp, syp, nb<I>(g, x, y, z, 0, -1, 1), sym, pe.cnu[1], acc, sh, kStapleReuse, 0);
    }
    Mat<T> u, w;
    load_link_r<R>(in.U, S, mu, s, u);
    mul_nn_traceless(u, acc, w);
    Alg<T> force, e;
    retr_itg(w, pick3(pe.gc, mu), force);
    load_alg(in.E, S, mu * 8, s, e);
#pragma unroll
    for (int a = 0; a < 8; a++) e.a[a] += force.a[a];
    if (mu == 2) {
      Alg<T> jp, jm;
      load_alg(in.Jp, S, 0, s, jp);
      load_alg(in.Jm, S, 0, s, jm);
#pragma unroll
      for (int a = 0; a < 8; a++) e.a[a] += pe.jz * (jp.a[a] - jm.a[a]);
    }
    if (!dry) {
      store_alg(in.E, S, mu * 8, s, e);
      if (sg >= 0) store_alg(in.E, S, mu * 8, sg, e);
    }
    LinkStep<T> X;
    Mat<T> uh;
    if (!pl.save_uold && mu != 2) {  // one exp at twice the angle, as in links_site
      X.set(T(2) * pick3(pl.cU, mu), e);
      X.apply(u, w);
      if (!dry) {
        store_link_r<R>(out.U, S, mu, s, w);
        if (sg >= 0) store_link_r<R>(out.U, S, mu, sg, w);
      }
      continue;
    }
    X.set(pick3(pl.cU, mu), e);
    X.apply(u, uh);
    if (pl.save_uold && !dry) {
      store_link(in.UOld, S, mu, s, uh);
      if (sg >= 0) store_link(in.UOld, S, mu, sg, uh);
    }
    X.apply(uh, w);
    if (!dry) {
      store_link_r<R>(out.U, S, mu, s, w);
      if (sg >= 0) store_link_r<R>(out.U, S, mu, sg, w);
    }
    if (mu == 2) fused_currents<T, I, R>(in, out, S, plane, s, sg, hi, u, uh, pl.cj, dry);
  }
}

}  // namespace glasma
