// observables.cu -- volume and per-slice reductions of the measurement path.
//
//   bulk       Observables::Bulk::Update (S/OBSERVABLES/BulkObservables.cpp:65-183):
//              sum_x 4 ReTr(1 - P_jk) per plane, sum_x E_mu^2, sum_x E_z (Jp-Jm)/sqrt2
//   gauss      GaussLaw::UpdateViolation (S/OBSERVABLES/GaussLawViolation.cpp:16-124) with
//              COMPUTE_GAUSS_VIOLATION (S/CALC/GaussViolation.cpp:13-23): max |G^a|, sum G^2 and
//              the per-z profile sum_{x,y,a} G^2 / (Nx Ny)
//   unitarity  Unitarity::UpdateViolation (S/OBSERVABLES/UnitarityViolation.cpp:13-51)
//   emt map    EnergyMomentumTensor::CreateMap (S/OBSERVABLES/EnergyMomentumTensor.cpp:92-170) with
//              COMPUTE_AVG_FIELD_STRENGTH (S/CALC/AvgFieldStrength.cpp:68-112)
//
// Every reduction is two-pass and deterministic: a fixed grid writes FP64 block partials
// (warp shuffles, then shared memory), a one-block pass sums them in a fixed order.
// Site arithmetic runs in FP64 accuracy: the matrix products in fixed point on the integer pipe (fx.cuh), or in FP64, out of
// line, where that does not hold the links.  The magnetic term of the bulk energy on FP32 lattices uses the identity
//   3 - ReTr(a b c^d d^d) = 1/2 ||A - B||^2 - 1/2 (n(a) + n(b) + n(c) + n(d)),
//   A = a b, B = d c, n(u) = ||u||_F^2 - 3  (zero for unitary u),
// exact with n(A) + n(B) in place of the four link terms and equal to it to first order in the links'
// departure from unitarity (~1e-7 for FP32-rounded links, so the difference is ~1e-14); the link
// terms are preferred because the products' own FP32 rounding never enters them:
// A, B and ||A - B||^2 are formed in FP32, whose rounding then costs about 1e-7 ||A - B|| per
// plaquette instead of 1e-7 (no cancellation against 3, so weak fields keep their digits), and the
// norm terms are summed in FP64 per link (each link's n counted for the plaquettes it belongs to).
#include <type_traits>

#include "fx.cuh"
#include "lattice.cuh"

namespace glasma {

namespace {

constexpr int kRedThreads = 256;
constexpr int kRedBlocks = 1216;  // 8 x 152 SMs
constexpr int kZChunks = 32;      // blocks per z slice for per-slice reductions

template <typename T>
__device__ __forceinline__ void load_link_d(const cx<T>* __restrict__ U, long long S, int mu, long long s, Mat<double>& m) {
  const cx<T>* p = U + (long long)(mu * 9) * S + s;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const cx<T> v = p[(long long)k * S];
    m.e[k] = mk<double>((double)v.re, (double)v.im);
  }
}
template <typename T>
__device__ __forceinline__ void load_alg_d(const T* __restrict__ F, long long S, long long base, long long s, Alg<double>& v) {
  const T* p = F + base * S + s;
#pragma unroll
  for (int a = 0; a < 8; a++) v.a[a] = (double)p[(long long)a * S];
}

__device__ __forceinline__ long long nbs(const Geometry& g, int x, int y, int z, int dx, int dy, int dz) {
  int xx = x + dx, yy = y + dy;
  xx = xx < 0 ? xx + g.nx : (xx >= g.nx ? xx - g.nx : xx);
  yy = yy < 0 ? yy + g.ny : (yy >= g.ny ? yy - g.ny : yy);
  return site_index(g, xx, yy, z + dz);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Block-reduce K values (the first KMAX of which are maxima when is_max[k]); thread 0 writes out[k].
template <int K>
__device__ __forceinline__ void block_reduce_store(double (&v)[K], const bool (&is_max)[K], double* out) {
  __shared__ double sh[K][kRedThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const double r = is_max[k] ? warp_max(v[k]) : warp_sum(v[k]);
    if (lane == 0) sh[k][warp] = r;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double r = (lane < (int)(blockDim.x / 32)) ? sh[k][lane] : 0.0;  // all reduced values are >= 0 or sums
      r = is_max[k] ? warp_max(r) : warp_sum(r);
      if (lane == 0) out[k] = r;
    }
  }
}

// Sum (or max) partials[b*K + k] over b in a fixed order; one block.
template <int K>
__global__ void finish_kernel(const double* __restrict__ partials, int nblocks, unsigned max_mask, double* out) {
  double v[K];
  bool is_max[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    v[k] = 0.0;
    is_max[k] = (max_mask >> k) & 1u;
  }
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < K; k++) {
      const double x = partials[(long long)b * K + k];
      v[k] = is_max[k] ? fmax(v[k], x) : v[k] + x;
    }
  block_reduce_store<K>(v, is_max, out);
}

// Per-slice finish: out[z*K + k] = sum_c partials[(z*kZChunks + c)*K + k] (max for masked k).  The sum carries its rounding
// errors along (two-sum): up to kZChunks equal parts one after the other would cost more digits than all that was summed
// before them (1.1e-16 rms over 18 parts, 1.5e-16 over 32).  Blocks of one warp: its ~200 FP64 instructions would queue for one
// SM's FP64 pipe (256 slices, ten sums: 11 us, 19 in blocks of 256 threads).
template <int K>
__global__ void finish_slices_kernel(const double* __restrict__ partials, int nz, unsigned max_mask, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nz * K) return;
  const int z = i / K, k = i - z * K;
  const double* p = partials + (long long)z * kZChunks * K + k;
  double v = 0.0, lost = 0.0;
  if ((max_mask >> k) & 1u) {
    for (int c = 0; c < kZChunks; c++) v = fmax(v, p[c * K]);
  } else {
#pragma unroll
    for (int c = 0; c < kZChunks; c++) {
      const double x = p[c * K], t = v + x, xx = t - v;
      lost += (v - (t - xx)) + (x - xx);
      v = t;
    }
  }
  out[i] = isfinite(lost) ? v + lost : v;  // an infinite sum has no remainder
}

// Index decodes in 32-bit arithmetic whenever the indices fit: GB300 runs the 64-bit integer
// division sequence partly on its FP64 pipe (measured on the gauge fixer's FP32 kernels), the pipe
// the FP64 observables are bound by.
__device__ __forceinline__ void decode_vol(const Geometry& g, long long idx, int& x, int& y, int& z) {
  if (g.vol < (1LL << 31)) {
    const unsigned u = (unsigned)idx, r = u / (unsigned)g.nx;
    x = (int)(u - r * (unsigned)g.nx);
    z = (int)(r / (unsigned)g.ny);
    y = (int)(r - (unsigned)z * (unsigned)g.ny);
    return;
  }
  const long long r = idx / g.nx;
  x = (int)(idx - r * g.nx);
  z = (int)(r / g.ny);
  y = (int)(r - (long long)z * g.ny);
}
// (x, y) of r = x + nx y within a transverse plane
__device__ __forceinline__ void decode_plane(const Geometry& g, long long r, int& x, int& y) {
  if (g.plane < (1LL << 31)) {
    const unsigned u = (unsigned)r;
    y = (int)(u / (unsigned)g.nx);
    x = (int)(u - (unsigned)y * (unsigned)g.nx);
    return;
  }
  y = (int)(r / g.nx);
  x = (int)(r - (long long)y * g.nx);
}

// Re tr(a b c^d d^d) = Re sum_ij (a b)_ij conj((d c)_ij): two products and a dot product instead of
// the three products of the full plaquette (the bulk energy needs only its trace)
__device__ __forceinline__ double retr_plaq(const Mat<double>& a, const Mat<double>& b, const Mat<double>& c,
                                           const Mat<double>& d) {
  Mat<double> A, B;
  mul_nn(a, b, A);
  mul_nn(d, c, B);
  double t = 0.0;
#pragma unroll
  for (int k = 0; k < 9; k++) t = fma(A.e[k].re, B.e[k].re, fma(A.e[k].im, B.e[k].im, t));
  return t;
}

// ||A - B||^2 of the plaquette a b (d c)^d in the (j,k) plane, A = U_j(x) U_k(x+j), B = U_k(x) U_j(x+k), FP32
__device__ __forceinline__ float plaq_sqdiff_f(const cx<float>* __restrict__ U, long long S, int j, int k,
                                               long long s, long long sj, long long sk) {
  Mat<float> a, b, A, B;
  load_link<float, long long>(U, S, j, s, a);
  load_link<float, long long>(U, S, k, sj, b);
  mul_nn(a, b, A);
  load_link<float, long long>(U, S, k, s, a);
  load_link<float, long long>(U, S, j, sk, b);
  mul_nn(a, b, B);
  float d2 = 0.f;
#pragma unroll
  for (int e = 0; e < 9; e++) {
    const float dr = A.e[e].re - B.e[e].re, di = A.e[e].im - B.e[e].im;
    d2 = fmaf(dr, dr, fmaf(di, di, d2));
  }
  return d2;
}

// n(u) = ||u||_F^2 - 3, in fixed point (fx.cuh: the squares to 2^-58, below FP64's rounding at 3) on the integer pipe:
// in FP64 its conversions and fmas bound the FP32 bulk energy
__device__ __noinline__ double link_norm_dev_fp64(const cx<float>* U, long long S, int mu, long long s) {
  const cx<float>* p = U + (long long)(mu * 9) * S + s;
  double n = -3.0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const cx<float> v = p[(long long)k * S];
    n = fma((double)v.re, (double)v.re, fma((double)v.im, (double)v.im, n));
  }
  return n;
}
__device__ __forceinline__ double link_norm_dev(const cx<float>* __restrict__ U, long long S, int mu, long long s) {
  const cx<float>* p = U + (long long)(mu * 9) * S + s;
  fx::Acc a = fx::acc_half();
  int top = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const cx<float> v = p[(long long)k * S];
    top = max(top, max(fx::habs(v.re), fx::habs(v.im)));
    const fx::R re = fx::to_fixed_split(fabsf(v.re), fx::shift(fx::kScale)), im = fx::to_fixed_split(fabsf(v.im), fx::shift(fx::kScale));
    fx::mad(a, re, re);
    fx::mad(a, im, im);
  }
  // Eighteen squares may add up to 19, beyond the format's +-8.  finish's 64-bit sum wraps there and is exact again after the
  // subtraction for norm^2 below 11; a.hh itself, 2^56 per unit, does not wrap.
  if (top > fx::kMaxEntryHi || (int)(a.hh >> 32) >= 10 << 24) return link_norm_dev_fp64(U, S, mu, s);
  return fx::from_fixed(fx::finish(a) - 3 * (1LL << fx::kScale), -fx::kScale);
}
// sum of squares of eight FP32 components, to 2^-58 of it
__device__ __forceinline__ double squares(const Alg<float>& e) {
  int top = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) top = max(top, fx::habs(e.a[k]));
  if (top >= 0x43100000 || top < ((1023 - 100) << 20)) {  // beyond 2^50 or below 2^-100: FP64
    double q = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) q = fma((double)e.a[k], (double)e.a[k], q);
    return q;
  }
  const int em = fx::exponent_of(top) + 1, sh = fx::shift(fx::kScale - em);
  fx::Acc a = fx::acc_half();
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const fx::R r = fx::to_fixed_split(fabsf(e.a[k]), sh);
    fx::mad(a, r, r);
  }
  return fx::from_fixed(fx::finish(a), 2 * em - fx::kScale);
}

// Site arithmetic of the FP64 sums on the integer pipe (fx.cuh): the magnetic terms are -Re tr(P - 1) from products of
// links held as U - 1 (nothing cancels against 3), the electric ones rotations.  What the fixed-point format does not
// hold goes through the FP64 forms, out of line.
constexpr int kFxThreads = 128;
constexpr int kFxMinBlocks = 3;     // 168 registers
constexpr int kFxBlocks = 912;      // grid-stride sums: two waves of 152 x 3

template <typename T>
__device__ __noinline__ double retr_plaq_fp64(const cx<T>* U, long long S, int p, int q, long long s, long long sp,
                                              long long sq) {
  Mat<double> a, b, c, d;
  load_link_d(U, S, p, s, a);
  load_link_d(U, S, q, sp, b);
  load_link_d(U, S, p, sq, c);
  load_link_d(U, S, q, s, d);
  return 3.0 - retr_plaq(a, b, c, d);
}
// 3 - Re tr of the plaquette (p, q) at s
template <typename T>
__device__ __forceinline__ double plaquette_defect(const cx<T>* __restrict__ U, long long S, int p, int q, long long s,
                                                   long long sp, long long sq) {
  fx::Guard guard = fx::guard_init();
  fx::M a, b, w, v;
  int ea, eb, ew, ev;
  fx::link_near(U, S, p, s, a, ea, guard);
  fx::link_near(U, S, q, sp, b, eb, guard);
  fx::near_product(a, ea, b, eb, w, ew, guard);
  fx::link_near(U, S, q, s, a, ea, guard);
  fx::link_near(U, S, p, sq, b, eb, guard);
  fx::near_product(a, ea, b, eb, v, ev, guard);
  if (fx::tripped(guard)) return retr_plaq_fp64(U, S, p, q, s, sp, sq);
  return fx::from_fixed(fx::plaquette_trace(w, ew, v, ev), max(ew, ev) - fx::kScale);
}
template <typename T>
__device__ __noinline__ void inv_adj_fp64(const cx<T>* U, const T* F, long long S, int mu, long long s, Alg<double>& out) {
  Mat<double> u;
  Alg<double> e;
  load_link_d(U, S, mu, s, u);
  load_alg_d(F, S, mu * 8, s, e);
  inv_adj_mul(u, e, out);
}
// U_mu^d(s) E_mu(s) U_mu(s)
template <typename T>
__device__ __forceinline__ void transported(const cx<T>* __restrict__ U, const T* __restrict__ E, long long S, int mu,
                                            long long s, const Alg<T>& e, Alg<double>& out) {
  fx::Guard guard = fx::guard_init();
  fx::M u, h;
  int eh;
  fx::ll o[8];
  fx::link_plain(U, S, mu, s, u, guard);
  fx::herm_one(e, h, eh, guard);
  fx::rotate_one(u, h, o, guard);
  fx::to_alg(o, eh - fx::kScale - 1, 1.0, out);
  if (fx::tripped(guard)) {
    Alg<double> t;
    inv_adj_fp64(U, E, S, mu, s, t);
    out = t;
  }
}

__global__ void __launch_bounds__(kFxThreads, kFxMinBlocks) bulk_fp64_kernel(Geometry g, FieldPtrs<double> f,
                                                                             double* partials) {
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  const bool is_max[7] = {false, false, false, false, false, false, false};
  const long long S = g.S;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < g.vol;
       idx += (long long)gridDim.x * blockDim.x) {
    int x, y, z;
    decode_vol(g, idx, x, y, z);
    const long long s = idx + g.plane;
#pragma unroll 1
    for (int n = 0; n < 3; n++) {  // planes (x,y), (x,z), (y,z)
      const int p = n == 2 ? 1 : 0, q = n == 0 ? 1 : 2;
      const long long sx = nbs(g, x, y, z, 1, 0, 0), sy = nbs(g, x, y, z, 0, 1, 0), sz = s + g.plane;
      const double m = 4.0 * plaquette_defect(f.U, S, p, q, s, n == 2 ? sy : sx, n == 0 ? sy : sz);
      if (n == 0)
        v[2] += m;
      else if (n == 1)
        v[1] += m;
      else
        v[0] += m;
    }
    for (int mu = 0; mu < 3; mu++) {
      Alg<double> e;
      load_alg_d(f.E, S, mu * 8, s, e);
      double q = 0.0;
#pragma unroll
      for (int k = 0; k < 8; k++) q += e.a[k] * e.a[k];
      v[3 + mu] += q;
      if (mu == 2) {
        Alg<double> jp, jm;
        load_alg_d(f.Jp, S, 0, s, jp);
        load_alg_d(f.Jm, S, 0, s, jm);
        double w = 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) w += e.a[k] * (jp.a[k] - jm.a[k]);
        v[6] += w * 0.70710678118654752440084436210484903928483593768847;
      }
    }
  }
  block_reduce_store<7>(v, is_max, partials + (long long)blockIdx.x * 7);
}

// The energies of an FP32 lattice (magnetic terms by the identity above).
__global__ void __launch_bounds__(kRedThreads) bulk_kernel(Geometry g, FieldPtrs<float> f, double* partials) {
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  const bool is_max[7] = {false, false, false, false, false, false, false};
  const long long S = g.S;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < g.vol;
       idx += (long long)gridDim.x * blockDim.x) {
    int x, y, z;
    decode_vol(g, idx, x, y, z);
    const long long s = idx + g.plane;
    const long long sxp = nbs(g, x, y, z, 1, 0, 0), syp = nbs(g, x, y, z, 0, 1, 0), szp = s + g.plane;
    // 4 (3 - ReTr P) = 2 ||A - B||^2 - 2 (n(a) + n(b) + n(c) + n(d)).  Summed over the lattice, a
    // plane with two periodic directions counts each of its links twice; in the planes with z
    // (open), the transverse link counts once at slice 0 and once more on the top ghost slice.
    const double nx = link_norm_dev(f.U, S, 0, s), ny = link_norm_dev(f.U, S, 1, s), nz = link_norm_dev(f.U, S, 2, s);
    const double wz = (z == 0) ? 1.0 : 2.0;
    double gx = 0.0, gy = 0.0;
    if (z == g.nz - 1) {
      gx = link_norm_dev(f.U, S, 0, szp);
      gy = link_norm_dev(f.U, S, 1, szp);
    }
    v[2] += 2.0 * (double)plaq_sqdiff_f(f.U, S, 0, 1, s, sxp, syp) - 2.0 * (2.0 * nx + 2.0 * ny);
    v[0] += 2.0 * (double)plaq_sqdiff_f(f.U, S, 1, 2, s, syp, szp) - 2.0 * (2.0 * nz + wz * ny + gy);
    v[1] += 2.0 * (double)plaq_sqdiff_f(f.U, S, 2, 0, s, szp, sxp) - 2.0 * (2.0 * nz + wz * nx + gx);
    for (int mu = 0; mu < 3; mu++) {
      Alg<float> e;
      load_alg<float, long long>(f.E, S, mu * 8, s, e);
      v[3 + mu] += squares(e);
      if (mu == 2) {
        Alg<float> jp, jm;
        load_alg<float, long long>(f.Jp, S, 0, s, jp);
        load_alg<float, long long>(f.Jm, S, 0, s, jm);
        double w = 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) w += (double)e.a[k] * ((double)jp.a[k] - (double)jm.a[k]);
        v[6] += w * 0.70710678118654752440084436210484903928483593768847;
      }
    }
  }
  block_reduce_store<7>(v, is_max, partials + (long long)blockIdx.x * 7);
}

// Gauss law, per slice: grid (kZChunks, nz).  Partials per (z, chunk): {sum G^2, max |G|}.
template <typename T>
__global__ void __launch_bounds__(kFxThreads, kFxMinBlocks) gauss_kernel(Geometry g, FieldPtrs<T> f, double norm, double* partials) {
  double v[2] = {0.0, 0.0};
  const bool is_max[2] = {false, true};
  const int z = blockIdx.y;
  const long long S = g.S;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < g.plane; r += (long long)gridDim.x * blockDim.x) {
    int x, y;
    decode_plane(g, r, x, y);
    const long long s = site_index(g, x, y, z);
    Alg<double> tot;
#pragma unroll
    for (int a = 0; a < 8; a++) tot.a[a] = 0.0;
#pragma unroll 1
    for (int mu = 0; mu < 3; mu++) {
      const long long sb = mu == 0 ? nbs(g, x, y, z, -1, 0, 0) : (mu == 1 ? nbs(g, x, y, z, 0, -1, 0) : s - g.plane);
      Alg<T> em;
      Alg<double> e, down;
      load_alg<T, long long>(f.E, S, mu * 8, sb, em);
      transported(f.U, f.E, S, mu, sb, em, down);
      load_alg_d(f.E, S, mu * 8, s, e);
#pragma unroll
      for (int a = 0; a < 8; a++) tot.a[a] += (e.a[a] - down.a[a]);
    }
    Alg<double> jp, jm;
    load_alg_d(f.JpStat, S, 0, s, jp);
    load_alg_d(f.JmStat, S, 0, s, jm);
#pragma unroll
    for (int a = 0; a < 8; a++) {
      const double G = norm * (tot.a[a] - (jp.a[a] + jm.a[a]) * 0.70710678118654752440084436210484903928483593768847);
      v[0] += G * G;
      v[1] = fmax(v[1], fabs(G));
    }
  }
  block_reduce_store<2>(v, is_max, partials + ((long long)z * kZChunks + blockIdx.x) * 2);
}

// ||U U^d - 1||_F^2
template <typename T>
__device__ __forceinline__ double unitarity_direct(const cx<T>* U, long long S, int mu, long long s) {
  Mat<double> u;
  load_link_d(U, S, mu, s, u);
  const double n = unitarity_norm(u);
  return n * n;
}
template <typename T>
__device__ __noinline__ double unitarity_far(const cx<T>* U, long long S, int mu, long long s) {
  return unitarity_direct(U, S, mu, s);
}
// FP32 links: U U^d - 1 and the sum of its squares in fixed point (2^-58 beside deviations of ~1e-7), where FP64 kept the FP64
// pipe busy with the 18 conversions and 54 products a link needs.  96x80x250: 1.50 ms in FP64, 0.26 here.  FP64 links deviate by
// rounding only, and stay in FP64.
__device__ __forceinline__ double unitarity_fx(const cx<float>* U, long long S, int mu, long long s) {
  fx::Guard g = fx::guard_init();
  fx::M m;
  fx::link_plain(U, S, mu, s, m, g);
  fx::R nI[9];
#pragma unroll
  for (int k = 0; k < 9; k++) nI[k] = fx::neg(m.e[k].im);
  fx::ll d[9];  // the diagonal, then the real and imaginary parts above it
  int n = 3;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = i; j < 3; j++) {
      fx::Acc a = fx::acc_half(), b = fx::acc_half();
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const fx::C &p = m.e[i + 3 * k], &q = m.e[j + 3 * k];
        fx::mad(a, p.re, q.re);
        fx::mad(a, p.im, q.im);
        if (i != j) {
          fx::mad(b, p.im, q.re);
          fx::mad(b, p.re, nI[j + 3 * k]);
        }
      }
      if (i == j) {
        d[i] = fx::finish(a) - (1LL << fx::kScale);
      } else {
        d[n++] = fx::finish(a);
        d[n++] = fx::finish(b);
      }
    }
  unsigned long long any = 0;
#pragma unroll
  for (int k = 0; k < 9; k++) any |= (unsigned long long)(d[k] ^ (d[k] >> 63));
  const int up = __clzll((long long)any) - 4;  // |d| 2^up < 2^60
  fx::Acc diag = fx::acc_half(), off = fx::acc_half();
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const fx::ll t = up >= 0 ? d[k] << up : d[k] >> -up;
    const fx::R r = fx::split((t ^ (t >> 63)) - (t >> 63));
    fx::mad(k < 3 ? diag : off, r, r);
  }
  if (fx::tripped(g)) return unitarity_far(U, S, mu, s);
  // six squares of off-diagonal numbers count twice
  return fx::from_fixed(fx::finish(diag), -2 * up - fx::kScale) + fx::from_fixed(fx::finish(off), 1 - 2 * up - fx::kScale);
}
__device__ __forceinline__ double unitarity_of(const cx<float>* U, long long S, int mu, long long s) {
  return unitarity_fx(U, S, mu, s);
}
__device__ __forceinline__ double unitarity_of(const cx<double>* U, long long S, int mu, long long s) {
  return unitarity_direct(U, S, mu, s);
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads) unitarity_kernel(Geometry g, const cx<T>* U, double* partials) {
  double v[2] = {0.0, 0.0};
  const bool is_max[2] = {false, true};
  const long long n = g.vol * 3;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int mu = i < g.vol ? 0 : (i < 2 * g.vol ? 1 : 2);
    const long long s = i - (long long)mu * g.vol + g.plane;
    const double n = unitarity_of(U, g.S, mu, s);
    v[0] += n;
    v[1] = fmax(v[1], n);
  }
  v[1] = sqrt(v[1]);
  block_reduce_store<2>(v, is_max, partials + (long long)blockIdx.x * 2);
}

__device__ __forceinline__ double dot8(const Alg<double>& p, const Alg<double>& q) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; k++) s += p.a[k] * q.a[k];
  return s;
}

// Clover average of the four plaquettes in plane (mu,nu) around x, as COMPUTE_AVG_MAGNETIC_FIELD_STRENGTH
// builds it from the elementary, neighbouring and extended plaquettes (S/CALC/Plaquettes.cpp:83-103).
template <typename T>
__device__ void clover(const Geometry& g, const cx<T>* U, int x, int y, int z, int mu, int nu, Mat<double>& avg) {
  const long long S = g.S;
  int dmu[3] = {0, 0, 0}, dnu[3] = {0, 0, 0};
  dmu[mu] = 1;
  dnu[nu] = 1;
  auto at = [&](int amu, int anu) { return nbs(g, x, y, z, amu * dmu[0] + anu * dnu[0], amu * dmu[1] + anu * dnu[1], amu * dmu[2] + anu * dnu[2]); };
  Mat<double> a, b, c, d, t1, t2, P;
  set_zero(avg);
  // elementary U_{mu nu}(x) = U_mu(x) U_nu(x+mu) U_mu^d(x+nu) U_nu^d(x)            (UUDD)
  load_link_d(U, S, mu, at(0, 0), a);
  load_link_d(U, S, nu, at(1, 0), b);
  load_link_d(U, S, mu, at(0, 1), c);
  load_link_d(U, S, nu, at(0, 0), d);
  mul_nn(a, b, t1);
  mul_dd(c, d, t2);
  mul_nn(t1, t2, P);
  for (int k = 0; k < 9; k++) { avg.e[k].re += P.e[k].re; avg.e[k].im += P.e[k].im; }
  // U_{-mu nu}(x) = U_nu(x) U_mu^d(x+nu-mu) U_nu^d(x-mu) U_mu(x-mu)                    (UDDU)
  load_link_d(U, S, nu, at(0, 0), a);
  load_link_d(U, S, mu, at(-1, 1), b);
  load_link_d(U, S, nu, at(-1, 0), c);
  load_link_d(U, S, mu, at(-1, 0), d);
  mul_nd(a, b, t1);
  mul_dn(c, d, t2);
  mul_nn(t1, t2, P);
  for (int k = 0; k < 9; k++) { avg.e[k].re += P.e[k].re; avg.e[k].im += P.e[k].im; }
  // U_{mu -nu}(x) = U_nu^d(x-nu) U_mu(x-nu) U_nu(x-nu+mu) U_mu^d(x)                    (DUUD)
  load_link_d(U, S, nu, at(0, -1), a);
  load_link_d(U, S, mu, at(0, -1), b);
  load_link_d(U, S, nu, at(1, -1), c);
  load_link_d(U, S, mu, at(0, 0), d);
  mul_dn(a, b, t1);
  mul_nd(c, d, t2);
  mul_nn(t1, t2, P);
  for (int k = 0; k < 9; k++) { avg.e[k].re += P.e[k].re; avg.e[k].im += P.e[k].im; }
  // U_{-mu -nu}(x) = U_mu^d(x-mu) U_nu^d(x-mu-nu) U_mu(x-mu-nu) U_nu(x-nu)             (DDUU)
  load_link_d(U, S, mu, at(-1, 0), a);
  load_link_d(U, S, nu, at(-1, -1), b);
  load_link_d(U, S, mu, at(-1, -1), c);
  load_link_d(U, S, nu, at(0, -1), d);
  mul_dd(a, b, t1);
  mul_nn(c, d, t2);
  mul_nn(t1, t2, P);
  for (int k = 0; k < 9; k++) { avg.e[k].re += P.e[k].re; avg.e[k].im += P.e[k].im; }
  for (int k = 0; k < 9; k++) { avg.e[k].re *= 0.25; avg.e[k].im *= 0.25; }
}

// The clover average in fixed point, one leaf at a time: leaf = W V^d with W, V products of two links or daggers,
//   U_mu(x) U_nu(x+mu)         | U_nu(x) U_mu(x+nu)
//   U_nu(x) U_mu^d(x-mu+nu)    | U_mu^d(x-mu) U_nu(x-mu)
//   U_nu^d(x-nu) U_mu(x-nu)    | U_mu(x) U_nu^d(x-nu+mu)
//   U_mu^d(x-mu) U_nu^d(x-mu-nu) | U_nu^d(x-nu) U_mu^d(x-mu-nu)
// B = 2 ReTr(i t avg), defect = 4 (3 - Re tr avg).  The leaves' own links are multiplied, no U U^d = 1 is used (FP32
// links satisfy it to 1e-7 only).
template <typename T>
__device__ __noinline__ void clover_fp64(const Geometry& g, const cx<T>* U, int x, int y, int z, int mu, int nu,
                                         Alg<double>& B, double& defect) {
  Mat<double> avg;
  clover(g, U, x, y, z, mu, nu, avg);
  retr_itg(avg, 2.0, B);
  defect = 4.0 * (3.0 - avg.e[0].re - avg.e[4].re - avg.e[8].re);
}
template <typename T>
__device__ __forceinline__ void clover_fx(const Geometry& g, const cx<T>* __restrict__ U, int x, int y, int z, int mu,
                                          int nu, Alg<double>& B, double& defect) {
  const long long S = g.S;
  auto at = [&](int m, int n) {
    const int d0 = (mu == 0 ? m : 0) + (nu == 0 ? n : 0), d1 = (mu == 1 ? m : 0) + (nu == 1 ? n : 0),
              d2 = (mu == 2 ? m : 0) + (nu == 2 ? n : 0);
    return nbs(g, x, y, z, d0, d1, d2);
  };
  fx::Guard guard = fx::guard_init();
#pragma unroll
  for (int k = 0; k < 8; k++) B.a[k] = 0.0;
  defect = 0.0;
#pragma unroll 1
  for (int l = 0; l < 4; l++) {
    // the leaf's lower corner c = x + lm mu + ln nu: its mu links are at c and c + nu, its nu links at c and c + mu
    const int lm = (l & 1) ? -1 : 0, ln = l >= 2 ? -1 : 0;
    const long long c = at(lm, ln), cm = at(lm + 1, ln), cn = at(lm, ln + 1);
    fx::M w, v;
    int ew, ev;
    // W, then V, by one copy of the code (with two the kernel waits for instructions: 64x64x256 FP64 4.66 ms for 4.61)
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
      const bool mu_up = ((l & 1) ^ h) != 0, nu_up = (l < 2) != (h != 0), swap = (l == 1 || l == 2) != (h != 0);
      const long long s_mu = mu_up ? cn : c, s_nu = nu_up ? cm : c;
      fx::M a, b;
      int ea, eb;
      if (h) {
        w = v;
        ew = ev;
      }
      fx::link_near(U, S, swap ? nu : mu, swap ? s_nu : s_mu, a, ea, guard, swap ? l >= 2 : (l & 1) != 0);
      fx::link_near(U, S, swap ? mu : nu, swap ? s_mu : s_nu, b, eb, guard, swap ? (l & 1) != 0 : l >= 2);
      fx::near_product(a, ea, b, eb, v, ev, guard);
    }
    fx::Anti p;
    fx::plaquette_parts(w, ew, v, ev, p);
#pragma unroll
    for (int k = 0; k < 8; k++) B.a[k] += fx::from_fixed(fx::component(p, k), p.e - fx::kScale);
    defect += fx::from_fixed(fx::plaquette_trace(w, ew, v, ev), p.e - fx::kScale);
  }
#pragma unroll
  for (int k = 0; k < 8; k++) B.a[k] *= k == 7 ? -0.25 * Consts<double>::inv_sqrt3() : -0.25;
  if (fx::tripped(guard)) {
    Alg<double> t;
    double d;
    clover_fp64(g, U, x, y, z, mu, nu, t, d);
    B = t;
    defect = d;
  }
}

// Energy-momentum tensor map, grid (kZChunks, nz); partials per (z, chunk): 10 sums.
template <typename T>
__global__ void __launch_bounds__(kFxThreads, kFxMinBlocks) emt_kernel(Geometry g, FieldPtrs<T> f, double aScale, double* partials) {
  double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  const bool is_max[10] = {false, false, false, false, false, false, false, false, false, false};
  const int z = blockIdx.y;
  const long long S = g.S;
  const double a3 = g.a[0] * g.a[1] * g.a[2];
  double q[3];
  for (int mu = 0; mu < 3; mu++) q[mu] = g.a[mu] * aScale * aScale / a3;
  const double inv = 1.0 / ((double)g.nx * g.ny);
  // the site's B waits in shared memory: held in registers through the transports it would spill
  __shared__ double sB[24 * kFxThreads];
  double* const tb = sB + threadIdx.x;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < g.plane; r += (long long)gridDim.x * blockDim.x) {
    int x, y;
    decode_plane(g, r, x, y);
    const long long s = site_index(g, x, y, z);
    // magnetic: clover averages of UOld in the planes yz (B0), zx (B1), xy (B2)
    double Bs[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int i = 0; i < 3; i++) {
      Alg<double> b;
      double d;
      clover_fx(g, f.UOld, x, y, z, i == 2 ? 0 : i + 1, i == 0 ? 2 : i - 1, b, d);
#pragma unroll
      for (int k = 0; k < 8; k++) tb[(i * 8 + k) * kFxThreads] = b.a[k];
      Bs[0] = i == 0 ? d : Bs[0];
      Bs[1] = i == 1 ? d : Bs[1];
      Bs[2] = i == 2 ? d : Bs[2];
    }
    // electric: average with the parallel-transported backward neighbour, using U
    Alg<double> Ev[3];
    double Es[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int mu = 0; mu < 3; mu++) {
      const long long sb = mu == 0 ? nbs(g, x, y, z, -1, 0, 0) : (mu == 1 ? nbs(g, x, y, z, 0, -1, 0) : s - g.plane);
      Alg<T> em;
      Alg<double> e, down;
      load_alg<T, long long>(f.E, S, mu * 8, sb, em);
      transported(f.U, f.E, S, mu, sb, em, down);
      load_alg_d(f.E, S, mu * 8, s, e);
      double sq = 0.0;
#pragma unroll
      for (int a = 0; a < 8; a++) {
        down.a[a] = 0.5 * (e.a[a] + down.a[a]);
        sq += 0.5 * (e.a[a] * e.a[a] + (double)em.a[a] * (double)em.a[a]);
      }
#pragma unroll
      for (int n = 0; n < 3; n++)  // by selection: an index would move the array to local memory
        if (n == mu) {
          Ev[n] = down;
          Es[n] = sq;
        }
    }
    Alg<double> B[3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int k = 0; k < 8; k++) B[i].a[k] = tb[(i * 8 + k) * kFxThreads];
    const double e0 = q[0] * q[0] * Es[0], e1 = q[1] * q[1] * Es[1], e2 = q[2] * q[2] * Es[2];
    const double b0 = q[0] * q[0] * Bs[0], b1 = q[1] * q[1] * Bs[1], b2 = q[2] * q[2] * Bs[2];
    v[0] += (0.5 * (e0 + e1 + e2 + b0 + b1 + b2)) * inv;
    v[1] += (0.5 * ((e1 + e2 + b1 + b2) - (e0 + b0))) * inv;
    v[2] += (0.5 * ((e0 + e2 + b0 + b2) - (e1 + b1))) * inv;
    v[3] += (0.5 * ((e0 + e1 + b0 + b1) - (e2 + b2))) * inv;
    v[4] += (q[1] * q[2] * dot8(Ev[1], B[2]) - q[2] * q[1] * dot8(Ev[2], B[1])) * inv;
    v[5] += (q[2] * q[0] * dot8(Ev[2], B[0]) - q[0] * q[2] * dot8(Ev[0], B[2])) * inv;
    v[6] += (q[0] * q[1] * dot8(Ev[0], B[1]) - q[1] * q[0] * dot8(Ev[1], B[0])) * inv;
    v[7] += (q[0] * q[1] * dot8(Ev[0], Ev[1]) + q[0] * q[1] * dot8(B[0], B[1])) * inv;
    v[8] += (q[1] * q[2] * dot8(Ev[1], Ev[2]) + q[1] * q[2] * dot8(B[1], B[2])) * inv;
    v[9] += (q[2] * q[0] * dot8(Ev[2], Ev[0]) + q[2] * q[0] * dot8(B[2], B[0])) * inv;
  }
  block_reduce_store<10>(v, is_max, partials + ((long long)z * kZChunks + blockIdx.x) * 10);
}

// zprofile[z] = slices[2z] / (Nx Ny)
__global__ void profile_scale_kernel(const double* sl, int nz, double inv, double* out) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  if (z < nz) out[z] = sl[2 * z] * inv;
}

}  // namespace

long long observable_scratch_doubles(const Geometry& g) {
  long long a = (long long)kRedBlocks * 8;
  long long b = (long long)g.nz * kZChunks * 10 + (long long)g.nz * 10;
  return (a > b ? a : b) + 64;
}

static unsigned red_blocks(long long n) {
  long long b = (n + kRedThreads - 1) / kRedThreads;
  return (unsigned)(b < kRedBlocks ? (b < 1 ? 1 : b) : kRedBlocks);
}

template <typename T>
cudaError_t launch_bulk(const Geometry& g, FieldPtrs<T> f, double* partials, double* result7, cudaStream_t stream) {
  unsigned nb;
  if constexpr (std::is_same<T, double>::value) {
    const long long n = (g.vol + kFxThreads - 1) / kFxThreads;
    nb = (unsigned)(n < kFxBlocks ? n : kFxBlocks);
    bulk_fp64_kernel<<<nb, kFxThreads, 0, stream>>>(g, f, partials);
  } else {
    nb = red_blocks(g.vol);
    bulk_kernel<<<nb, kRedThreads, 0, stream>>>(g, f, partials);
  }
  finish_kernel<7><<<1, kRedThreads, 0, stream>>>(partials, (int)nb, 0u, result7);
  return cudaGetLastError();
}

// result2 = {sum G^2, max|G|}; zprofile (device, may be null) = per-slice sum G^2 / (Nx Ny)
template <typename T>
cudaError_t launch_gauss(const Geometry& g, FieldPtrs<T> f, double a_scale, double* partials, double* result2,
                         double* zprofile, cudaStream_t stream) {
  const double norm = a_scale * a_scale * a_scale / (g.a[0] * g.a[1] * g.a[2]);
  dim3 grid(kZChunks, g.nz);
  gauss_kernel<T><<<grid, kFxThreads, 0, stream>>>(g, f, norm, partials);
  double* slices = partials + (long long)g.nz * kZChunks * 2;
  finish_slices_kernel<2><<<(g.nz * 2 + 31) / 32, 32, 0, stream>>>(partials, g.nz, 2u, slices);
  finish_kernel<2><<<1, kRedThreads, 0, stream>>>(slices, g.nz, 2u, result2);
  if (zprofile) {
    profile_scale_kernel<<<(g.nz + 255) / 256, 256, 0, stream>>>(slices, g.nz, 1.0 / ((double)g.nx * g.ny), zprofile);
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_unitarity(const Geometry& g, const cx<T>* U, double* partials, double* result2, cudaStream_t stream) {
  const unsigned nb = red_blocks(g.vol * 3);
  unitarity_kernel<T><<<nb, kRedThreads, 0, stream>>>(g, U, partials);
  finish_kernel<2><<<1, kRedThreads, 0, stream>>>(partials, (int)nb, 2u, result2);
  return cudaGetLastError();
}

// result (device) = Nz x 10
template <typename T>
cudaError_t launch_emt_map(const Geometry& g, FieldPtrs<T> f, double a_scale, double* partials, double* result,
                           cudaStream_t stream) {
  dim3 grid(kZChunks, g.nz);
  emt_kernel<T><<<grid, kFxThreads, 0, stream>>>(g, f, a_scale, partials);
  finish_slices_kernel<10><<<(g.nz * 10 + 31) / 32, 32, 0, stream>>>(partials, g.nz, 0u, result);
  return cudaGetLastError();
}

#define GLASMA_OBS_INSTANTIATE(T)                                                                               \
  template cudaError_t launch_bulk<T>(const Geometry&, FieldPtrs<T>, double*, double*, cudaStream_t);          \
  template cudaError_t launch_gauss<T>(const Geometry&, FieldPtrs<T>, double, double*, double*, double*,       \
                                       cudaStream_t);                                                           \
  template cudaError_t launch_unitarity<T>(const Geometry&, const cx<T>*, double*, double*, cudaStream_t);     \
  template cudaError_t launch_emt_map<T>(const Geometry&, FieldPtrs<T>, double, double*, double*, cudaStream_t);

GLASMA_OBS_INSTANTIATE(double)
GLASMA_OBS_INSTANTIATE(float)

}  // namespace glasma
