// fft.cuh -- batched 1D transforms of lengths 2^a 3^b 5^c: self-sorting mixed-radix (Stockham) passes with up to sixteen
// values of a line in a thread's registers.
//
// A block takes `tl` neighbouring lines.  The first stage reads its values from global memory straight into registers, the
// last writes them back from registers, and shared memory only carries the values between two stages: one round trip
// for the lengths up to 256 (16 x 16), two up to 4096, where the radix-2 passes it replaces made seven to nine.
// Stage with Ns = product of the earlier radices, butterfly j < n/R of a line:
//   v_r = in[j + r n/R] w^(r (j mod Ns) n/(Ns R)),  r < R            (w = exp(-+2 pi i / n))
//   out[(j / Ns) Ns R + (j mod Ns) + q Ns] = sum_r v_r exp(-+2 pi i r q / R),  q < R
// (e.g. Govindaraju et al., SC 2008).  The first stage has no twiddles.
//
// Bound: FP64 by the FP64 pipe (a radix-16 pass costs ~10 FP64 operations per element, a radix-2 pass 4), FP32 by
// latency and the round trips.
//
// kScale: the transform along z, the multiplication by 1 / (V p^2) and the inverse transform along z in one pass over
// the data (the acceleration step of the gauge fixer): two passes and a kernel fewer per iteration.
#pragma once

#include <cuda_runtime.h>

namespace glasma {
namespace fft {

struct Plan {
  int n;
  int nstages;
  int radix[12];
  unsigned magic[12];  // floor(j * magic / 2^32) = j / Ns for j < 2^16, Ns the product of the earlier radices
};

// the momentum factor of the acceleration step
template <typename Re>
struct Scale {
  int nx, ny;
  Re v;                  // sites
  const Re* tab;         // momenta per axis: nx, then ny, then nz
  int project_zero;
};

template <typename C>
struct Real;
template <>
struct Real<double2> {
  typedef double type;
};
template <>
struct Real<float2> {
  typedef float type;
};

__device__ __forceinline__ double2 make(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ float2 make(float x, float y) { return make_float2(x, y); }
template <typename C>
__device__ __forceinline__ C add(const C& a, const C& b) {
  return make(a.x + b.x, a.y + b.y);
}
template <typename C>
__device__ __forceinline__ C sub(const C& a, const C& b) {
  return make(a.x - b.x, a.y - b.y);
}
template <typename C>
__device__ __forceinline__ C mul(const C& a, const C& w) {
  return make(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
// -i z (forward), +i z (inverse)
template <bool kInv, typename C>
__device__ __forceinline__ C rot(const C& z) {
  return kInv ? make(-z.y, z.x) : make(z.y, -z.x);
}
// z times exp(-+2 pi i t) for t = (c, s) = (cos, sin) of 2 pi t
template <bool kInv, typename C, typename Re>
__device__ __forceinline__ C turn(const C& z, Re c, Re s) {
  return kInv ? make(z.x * c - z.y * s, z.y * c + z.x * s) : make(z.x * c + z.y * s, z.y * c - z.x * s);
}

template <bool kInv, typename C>
__device__ __forceinline__ void dft2(C& a, C& b) {
  const C t = a;
  a = add(t, b);
  b = sub(t, b);
}
template <bool kInv, typename C>
__device__ __forceinline__ void dft4(C& a, C& b, C& c, C& d) {
  const C s0 = add(a, c), d0 = sub(a, c), s1 = add(b, d), d1 = rot<kInv>(sub(b, d));
  a = add(s0, s1);
  b = add(d0, d1);
  c = sub(s0, s1);
  d = sub(d0, d1);
}
template <int R, bool kInv, typename C>
__device__ __forceinline__ void dft(C (&v)[R]) {
  typedef typename Real<C>::type Re;
  if constexpr (R == 2) {
    dft2<kInv>(v[0], v[1]);
  } else if constexpr (R == 4) {
    dft4<kInv>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 3) {
    const Re h = Re(0.86602540378443864676);  // sin(2 pi / 3)
    const C s = add(v[1], v[2]), f = sub(v[1], v[2]);
    const C m = make(v[0].x - Re(0.5) * s.x, v[0].y - Re(0.5) * s.y);
    const C d = rot<kInv>(make(h * f.x, h * f.y));
    v[0] = add(v[0], s);
    v[1] = add(m, d);
    v[2] = sub(m, d);
  } else if constexpr (R == 5) {
    const Re c1 = Re(0.30901699437494742410), c2 = Re(-0.80901699437494742410);  // cos(2 pi/5), cos(4 pi/5)
    const Re s1 = Re(0.95105651629515357212), s2 = Re(0.58778525229247312917);   // sin(2 pi/5), sin(4 pi/5)
    const C p1 = add(v[1], v[4]), m1 = sub(v[1], v[4]), p2 = add(v[2], v[3]), m2 = sub(v[2], v[3]);
    const C a1 = make(v[0].x + c1 * p1.x + c2 * p2.x, v[0].y + c1 * p1.y + c2 * p2.y);
    const C a2 = make(v[0].x + c2 * p1.x + c1 * p2.x, v[0].y + c2 * p1.y + c1 * p2.y);
    const C b1 = rot<kInv>(make(s1 * m1.x + s2 * m2.x, s1 * m1.y + s2 * m2.y));
    const C b2 = rot<kInv>(make(s2 * m1.x - s1 * m2.x, s2 * m1.y - s1 * m2.y));
    v[0] = make(v[0].x + p1.x + p2.x, v[0].y + p1.y + p2.y);
    v[1] = add(a1, b1);
    v[4] = sub(a1, b1);
    v[2] = add(a2, b2);
    v[3] = sub(a2, b2);
  } else if constexpr (R == 8) {
    const Re h = Re(0.70710678118654752440);
    dft4<kInv>(v[0], v[2], v[4], v[6]);
    dft4<kInv>(v[1], v[3], v[5], v[7]);
    const C o1 = turn<kInv>(v[3], h, h), o2 = rot<kInv>(v[5]), o3 = turn<kInv>(v[7], -h, h);
    const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = add(e0, o0);
    v[4] = sub(e0, o0);
    v[1] = add(e1, o1);
    v[5] = sub(e1, o1);
    v[2] = add(e2, o2);
    v[6] = sub(e2, o2);
    v[3] = add(e3, o3);
    v[7] = sub(e3, o3);
  } else {
    static_assert(R == 16, "radix");
    const Re h = Re(0.70710678118654752440), c = Re(0.92387953251128675613), s = Re(0.38268343236508977173);  // pi/8
#pragma unroll
    for (int b = 0; b < 4; b++) dft4<kInv>(v[b], v[b + 4], v[b + 8], v[b + 12]);
    // v[b + 4 k1] times w16^(b k1)
    v[5] = turn<kInv>(v[5], c, s);
    v[6] = turn<kInv>(v[6], h, h);
    v[7] = turn<kInv>(v[7], s, c);
    v[9] = turn<kInv>(v[9], h, h);
    v[10] = rot<kInv>(v[10]);
    v[11] = turn<kInv>(v[11], -h, h);
    v[13] = turn<kInv>(v[13], s, c);
    v[14] = turn<kInv>(v[14], -h, h);
    v[15] = turn<kInv>(v[15], -c, -s);
#pragma unroll
    for (int k = 0; k < 4; k++) dft4<kInv>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    // out[k1 + 4 k2] = v[4 k1 + k2]
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = a + 1; b < 4; b++) {
        const C t = v[4 * a + b];
        v[4 * a + b] = v[4 * b + a];
        v[4 * b + a] = t;
      }
  }
}

constexpr int kThreads = 256;  // most threads of a block

// Shared-memory position of element k of line t: consecutive lines next to each other for strided lines; a pad per 16
// elements where the lines are contiguous (a thread's outputs of the first stage are 16 apart).
template <bool kContig>
__device__ __forceinline__ int place(int t, int k, int pitch, int log_tl) {
  return kContig ? t * pitch + k + (k >> 4) : (k << log_tl) + t;
}
__host__ __device__ __forceinline__ int line_pitch(int n) { return n + (n >> 4) + 1; }

template <typename C, int R, bool kInv, bool kContig, typename Ld, typename St>
__device__ __forceinline__ void stage(int n, int Ns, unsigned magic, int tl, int log_tl, const C* __restrict__ tw,
                                      const Ld& ld, const St& st) {
  const int nb = n / R, tstep = nb / Ns;
  for (int idx = threadIdx.x; idx < tl * nb; idx += blockDim.x) {
    int t, j;
    if (kContig) {
      t = idx / nb;
      j = idx - t * nb;
    } else {
      t = idx & (tl - 1);
      j = idx >> log_tl;
    }
    C v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = ld(t, j + r * nb);
    const int jm = Ns == 1 ? 0 : j - (int)__umulhi((unsigned)j, magic) * Ns;
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) {
        C w = tw[r * jm * tstep];
        if (kInv) w.y = -w.y;
        v[r] = mul(v[r], w);
      }
    }
    dft<R, kInv>(v);
    const int o = (j - jm) * R + jm;
#pragma unroll
    for (int q = 0; q < R; q++) st(t, o + q * Ns, v[q]);
  }
}

template <typename C, bool kInv, bool kContig, typename Ld, typename St>
__device__ __forceinline__ void stage_of(int radix, int n, int Ns, unsigned magic, int tl, int log_tl,
                                         const C* __restrict__ tw, const Ld& ld, const St& st) {
  switch (radix) {
    case 16: stage<C, 16, kInv, kContig>(n, Ns, magic, tl, log_tl, tw, ld, st); break;
    case 8: stage<C, 8, kInv, kContig>(n, Ns, magic, tl, log_tl, tw, ld, st); break;
    case 5: stage<C, 5, kInv, kContig>(n, Ns, magic, tl, log_tl, tw, ld, st); break;
    case 4: stage<C, 4, kInv, kContig>(n, Ns, magic, tl, log_tl, tw, ld, st); break;
    case 3: stage<C, 3, kInv, kContig>(n, Ns, magic, tl, log_tl, tw, ld, st); break;
    default: stage<C, 2, kInv, kContig>(n, Ns, magic, tl, log_tl, tw, ld, st);
  }
}

// Lines of length n: contiguous (kContig: line l at l n) or with stride st (line (o, i) at o st n + i, i < st), `tl` lines
// per block, blocks_per_row blocks per row of st lines (the last one ragged).  kScale: forward, scale, inverse.
template <typename C, bool kInv, bool kContig, bool kScale>
__global__ void __launch_bounds__(kThreads, 2)
    lines_kernel(C* X, const __grid_constant__ Plan plan, long long nlines, long long st, int tl, int log_tl,
                 unsigned blocks_per_row, const C* __restrict__ tw, Scale<typename Real<C>::type> sc) {
  typedef typename Real<C>::type Re;
  extern __shared__ __align__(16) unsigned char fft_lines_smem[];
  const int n = plan.n, pitch = line_pitch(n);
  const int buffer = kContig ? tl * pitch : tl * n;
  // a stage writes to b; the second buffer is not there (nor touched) with two stages
  C* b = reinterpret_cast<C*>(fft_lines_smem);
  C* a = b + buffer;
  long long base, i0 = 0;
  int live;  // lines of this block
  if (kContig) {
    base = (long long)blockIdx.x * tl * n;
    const long long left = nlines - (long long)blockIdx.x * tl;
    live = left < tl ? (int)left : tl;
  } else {
    const unsigned o = blockIdx.x / blocks_per_row;
    i0 = (long long)(blockIdx.x - o * blocks_per_row) * tl;
    base = (long long)o * st * n + i0;
    live = st - i0 < tl ? (int)(st - i0) : tl;
  }
  auto global = [&](int t, int k) -> C* { return X + base + (kContig ? (long long)t * n + k : t + (long long)k * st); };
  const C zero = make(Re(0), Re(0));
  constexpr int kHalves = kScale ? 2 : 1;
  int done = 0;
  const int total = kHalves * plan.nstages;
#pragma unroll
  for (int half = 0; half < kHalves; half++) {
    int Ns = 1;
    for (int s = 0; s < plan.nstages; s++, done++) {
      const bool first = done == 0, last = done == total - 1, scale = kScale && half == 1 && s == 0;
      auto ld = [&](int t, int k) -> C {
        if (first) return t < live ? *global(t, k) : zero;
        C v = a[place<kContig>(t, k, pitch, log_tl)];
        if (scale) {
          const unsigned i = (unsigned)(i0 + t), y = i / (unsigned)sc.nx, x = i - y * (unsigned)sc.nx;
          const Re p2 = t < live ? sc.tab[x] + sc.tab[sc.nx + y] + sc.tab[sc.nx + sc.ny + k] : Re(1);
          if (p2 > Re(0)) {
            const Re f = Re(1) / (sc.v * p2);
            v.x *= f;
            v.y *= f;
          } else if (sc.project_zero) {
            v = zero;
          }
        }
        return v;
      };
      auto store = [&](int t, int k, const C& v) {
        if (!last)
          b[place<kContig>(t, k, pitch, log_tl)] = v;
        else if (t < live)
          *global(t, k) = v;
      };
      if (kScale ? half == 1 : kInv)
        stage_of<C, true, kContig>(plan.radix[s], n, Ns, plan.magic[s], tl, log_tl, tw, ld, store);
      else
        stage_of<C, false, kContig>(plan.radix[s], n, Ns, plan.magic[s], tl, log_tl, tw, ld, store);
      if (!last) __syncthreads();
      // what was just written is read next; the other buffer is free once every thread is past the barrier
      C* const t = a;
      a = b;
      b = t;
      Ns *= plan.radix[s];
    }
  }
}

inline bool make_plan(int n, Plan& p) {
  p = Plan{};
  p.n = n;
  if (n < 2 || n >= (1 << 16)) return false;  // at most ten stages (3^10)
  int twos = 0, m = n;
  while (m % 2 == 0) m /= 2, twos++;
  auto push = [&](int r) { p.radix[p.nstages++] = r; };
  // powers of two in as few stages as radices up to 16 allow, none of them below 4 where that can be helped
  int stages = (twos + 3) / 4;
  for (int left = twos; stages > 0; stages--) {
    const int k = (left + stages - 1) / stages;
    push(1 << k);
    left -= k;
  }
  while (m % 5 == 0) m /= 5, push(5);
  while (m % 3 == 0) m /= 3, push(3);
  if (m != 1) return false;
  unsigned ns = 1;
  for (int s = 0; s < p.nstages; s++) {
    p.magic[s] = ns == 1 ? 0u : (unsigned)((0x100000000ULL + ns - 1) / ns);
    ns *= (unsigned)p.radix[s];
  }
  return true;
}

struct Shape {
  int tl, log_tl, threads;
  size_t smem;
};
// Lines per block: sixteen neighbouring ones are full sectors for the strided passes; fewer where the buffers (two, or
// one between two stages) would leave less than three blocks on an SM.  False: one line does not fit.
inline bool make_shape(const Plan& p, bool contig, bool scale, size_t elem, long long lines, Shape& s) {
  const int buffers = (scale ? 2 * p.nstages : p.nstages) > 2 ? 2 : (p.nstages > 1 || scale ? 1 : 0);
  const size_t line = (size_t)buffers * (contig ? line_pitch(p.n) : p.n) * elem;
  const size_t most = 227 * 1024, good = 72 * 1024;
  if (line > most) return false;
  s.tl = 16;
  s.log_tl = 4;
  while (s.tl > 1 && ((size_t)s.tl * line > good || s.tl / 2 >= lines)) s.tl /= 2, s.log_tl--;
  s.smem = (size_t)s.tl * line;
  int work = s.tl * (p.n / p.radix[0]);
  work = (work + 31) / 32 * 32;
  s.threads = work < 64 ? 64 : (work > kThreads ? kThreads : work);
  return true;
}

template <typename C, bool kInv, bool kContig, bool kScale>
cudaError_t launch(C* X, const Plan& plan, const Shape& s, long long st, long long total, const C* tw,
                   const Scale<typename Real<C>::type>& sc, cudaStream_t stream) {
  auto* k = lines_kernel<C, kInv, kContig, kScale>;
  if (s.smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
    if (e != cudaSuccess) return e;
  }
  const long long nlines = total / plan.n;
  long long per_row = 1, blocks;
  if (kContig) {
    blocks = (nlines + s.tl - 1) / s.tl;
  } else {
    per_row = (st + s.tl - 1) / s.tl;
    blocks = nlines / st * per_row;
  }
  k<<<(unsigned)blocks, s.threads, s.smem, stream>>>(X, plan, nlines, st, s.tl, s.log_tl, (unsigned)per_row, tw, sc);
  return cudaGetLastError();
}

}  // namespace fft
}  // namespace glasma
