// adjoint.cu -- adjoint (reverse-mode) leapfrog: gradients of a late-time observable with respect
// to the initial electric field and the initial colour currents, in the lattice's precision (FP64 or FP32).
//
// No reference counterpart.  Method:
//   forward   nsteps of the ordinary leapfrog, storing the state every `checkpoint_every` steps;
//   objective L = N(q)/D(q), q = (e0,e1,e2,b0,b1,b2) slice sums over z in [z0,z1):
//             e_mu = cE_mu sum_x E_mu^2, b_i = cB_i sum_x 4 ReTr(1 - P_jk) (the bulk observables'
//             constants, S/OBSERVABLES/BulkObservables.cpp:22-97), N, D linear forms (D = 1 when its
//             coefficients are all zero).  P_L/P_T: N = (1,1,-1,1,1,-1), D = (0,0,1,0,0,1).
//   backward  for t = nsteps-1 .. 0: reconstruct the state at t from the state at t+1 by
//             time-reversed integration (the step is an exact composition of shears: the forward
//             kernels run with -dt, the links are rotated back by X^dagger), or reload the checkpoint
//             at t; then pull the cotangents back through the step's sub-steps in reverse order.
// Cotangent convention: the steps multiply links by elements of SU(3) from the left, so a link's cotangent is the algebra vector l
// with dL = l.d for U -> exp(i t.d) U (eight numbers; no E or current gradient sees what else a matrix cotangent has).  With c = a x b for
// c^k = f^klm a_l b_m:
//   W = A B            -> l_A += l_W,  l_B += InvAdj(A, l_W)
//   y = Adj(V, e)      -> l_V += y x l_y,  l_e += InvAdj(V, l_y)
//   y = InvAdj(V, e)   -> l_V += e x Adj(V, l_y),  l_e += Adj(V, l_y)
//   X = exp(i c t.e)   -> l_e += c sum_n (c e x)^n l_X / (n + 1)!, or the Cayley-Hamilton form's derivative for |c e| >= 1
// FP64 does this in fixed point on the integer pipe (fx.cuh), since one FP64 instruction costs GB300 as much as 60 FP32 ones.
// 32x32x64, 20 steps, FP64: 47.1 ms with matrix cotangents in FP64, 40.9 with algebra vectors, 20.9 in fixed point.
// Ghost slices are copies of the boundary slices, so cotangents that land on a ghost are added to
// the slice it copies.
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/glasma_gb300.h"
#include "handle.h"
#include "leapfrog_sites.cuh"

namespace {

thread_local std::string g_adj_error;
int afail(int st, const std::string& m) {
  g_adj_error = m;
  return st;
}

struct DevBuf {
  void* p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
  bool alloc(size_t bytes) { return cudaMalloc(&p, bytes) == cudaSuccess; }
};

// Makes the pages of a host array that is about to be overwritten present and writable, by MADV_POPULATE_WRITE (Linux 5.14;
// without it the copy faults them in itself): the array keeps its contents, whatever happens to the call afterwards, and a
// bad address is an error of madvise, not a signal.  (An atomic or of zero at each page also keeps them, but Arm reports its
// fault as a read first: two faults per page, a first pass over 180 MB 68 ms for 40.)  Memory of a device, which the copy
// refuses or takes, is left alone.
void populate_pages(double* p, size_t bytes) {
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (a.type != cudaMemoryTypeUnregistered && a.type != cudaMemoryTypeHost) return;
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), from = reinterpret_cast<uintptr_t>(p) & ~(page - 1);
  madvise(reinterpret_cast<void*>(from), reinterpret_cast<uintptr_t>(p) + bytes - from, MADV_POPULATE_WRITE);
}

double ratio(const double* num, const double* den, const double* q, double* Nout, double* Dout) {
  double N = 0.0, D = 0.0;
  bool has_den = false;
  for (int k = 0; k < 6; k++) {
    N += num[k] * q[k];
    D += den[k] * q[k];
    if (den[k] != 0.0) has_den = true;
  }
  if (!has_den) D = 1.0;
  *Nout = N;
  *Dout = D;
  return N / D;
}

}  // namespace

namespace glasma {
// The FP64 kernels' rotations, plaquettes and exponential pull-back in fixed point on the integer pipe (fx.cuh): true when
// its numbers held the operands.  FP32 has its own pipe and always answers false.
template <bool kAdj, typename R>
__device__ __forceinline__ bool fixed_rotated(const cx<R>* U, long long S, int mu, long long s, const Alg<R>& e, Alg<R>& o) {
  if constexpr (sizeof(R) == 8) {
    fx::Guard g = fx::guard_init();
    fx::M v, h;
    int eh;
    fx::ll q[8];
    fx::link_plain<kAdj>(U, S, mu, s, v, g);  // Adj(V) = InvAdj(V^d)
    fx::herm_one(e, h, eh, g);
    fx::rotate_one(v, h, q, g);
    fx::to_alg(q, eh - fx::kScale - 1, 1.0, o);
    return !fx::tripped(g);
  }
  return false;
}
template <bool kAdj, typename R>
__device__ __forceinline__ bool fixed_rotated_pair(const cx<R>* U, long long S, int mu, long long s, const Alg<R>& e1,
                                                   const Alg<R>& e2, Alg<R>& o1, Alg<R>& o2) {
  if constexpr (sizeof(R) == 8) {
    fx::Guard g = fx::guard_init();
    fx::M v;
    fx::link_plain(U, S, mu, s, v, g);
    fx::adj_pair<!kAdj>(v, e1, e2, o1, o2, g);
    return !fx::tripped(g);
  }
  return false;
}
template <typename R>
__device__ __forceinline__ bool fixed_plaquette(const cx<R>* U, long long S, int p, int q, long long sa, long long sb,
                                                long long sc, Mat<R>& h, Alg<R>& al) {
  if constexpr (sizeof(R) == 8) {
    fx::Guard g = fx::guard_init();
    fx::M a, b, w, v;
    int ea, eb, ew, ev;
    fx::link_near(U, S, p, sa, a, ea, g);
    fx::link_near(U, S, q, sb, b, eb, g);
    fx::near_product(a, ea, b, eb, w, ew, g);
    fx::link_near(U, S, q, sa, a, ea, g);
    fx::link_near(U, S, p, sc, b, eb, g);
    fx::near_product(a, ea, b, eb, v, ev, g);
    fx::Anti t;
    fx::plaquette_full(w, ew, v, ev, t, h);
#pragma unroll
    for (int k = 0; k < 8; k++)
      al.a[k] = fx::from_fixed(fx::component(t, k), t.e - fx::kScale) * (k == 7 ? -0.5 * Consts<double>::inv_sqrt3() : -0.5);
    return !fx::tripped(g);
  }
  return false;
}
template <typename R>
__device__ __forceinline__ bool fixed_series(const Alg<R>& q, const Alg<R>& l, int terms, const R* inv, Alg<R>& o) {
  if constexpr (sizeof(R) == 8) return fx::exp_series(q, l, terms, inv, o);
  return false;
}
template <typename R>
__device__ __forceinline__ bool fixed_cross(const Alg<R>& a, const Alg<R>& b, Alg<R>& o) {
  if constexpr (sizeof(R) == 8) return fx::cross(a, b, o);
  return false;
}
template <typename R>
__device__ __forceinline__ bool fixed_trace_with(const Mat<R>& h, const Alg<R>& n, Alg<R>& o) {
  if constexpr (sizeof(R) == 8) return fx::trace_with(h, n, o);
  return false;
}
// X = exp(i c t.e) and out = X^d u
template <typename R>
__device__ __forceinline__ bool fixed_step_back(R c, const Alg<R>& e, const Mat<R>& u, Mat<R>& x, Mat<R>& out) {
  if constexpr (sizeof(R) == 8) {
    fx::M X, D;
    int ex;
    if (!fx::near_exp(c, e, X, ex)) return false;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const fx::C& t = X.e[i + 3 * j];
        x.e[i + 3 * j] = mk<double>((i == j ? 1.0 : 0.0) + fx::from_fixed(fx::join(t.re), ex - fx::kScale),
                                    fx::from_fixed(fx::join(t.im), ex - fx::kScale));
        D.e[j + 3 * i].re = t.re;
        D.e[j + 3 * i].im = fx::neg(t.im);
      }
    return fx::add_product(D, ex, u, out);
  }
  return false;
}

namespace adj64 {
#define ADJ_REAL double
#include "adjoint_kernels.inc"
#undef ADJ_REAL
}  // namespace adj64
namespace adj32 {
#define ADJ_REAL float
#include "adjoint_kernels.inc"
#undef ADJ_REAL
}  // namespace adj32
}  // namespace glasma

extern "C" {

int glasma_objective(glasma_lattice* h, int z_begin, int z_end, const double* num, const double* den, double* value) {
  if (!h || !num || !den || !value) return afail(GLASMA_ERR_INVALID_ARGUMENT, "null argument");
  if (z_begin < 0 || z_end > h->g.nz || z_begin >= z_end) return afail(GLASMA_ERR_INVALID_ARGUMENT, "bad slice range");
  cudaSetDevice(h->device);
  DevBuf scratch;
  if (!scratch.alloc(sizeof(double) * 608 * 6)) return afail(GLASMA_ERR_OUT_OF_MEMORY, "scratch");
  double q[6], N, D;
  int st = h->precision == GLASMA_FP64 ? glasma::adj64::objective_q(h, z_begin, z_end, q, static_cast<double*>(scratch.p))
                                       : glasma::adj32::objective_q(h, z_begin, z_end, q, static_cast<double*>(scratch.p));
  if (st) return st;
  *value = ratio(num, den, q, &N, &D);
  return GLASMA_OK;
}

int glasma_adjoint(glasma_lattice* h, double dt, int nsteps, int checkpoint_every, int z_begin, int z_end,
                   const double* num, const double* den, double* objective, double* grad_E, double* grad_Jp,
                   double* grad_Jm, double* grad_JpStat, double* grad_JmStat) {
  if (!h || !num || !den) return afail(GLASMA_ERR_INVALID_ARGUMENT, "null argument");
  if (nsteps < 1 || checkpoint_every < 1) return afail(GLASMA_ERR_INVALID_ARGUMENT, "nsteps, checkpoint_every >= 1");
  if (z_begin < 0 || z_end > h->g.nz || z_begin >= z_end) return afail(GLASMA_ERR_INVALID_ARGUMENT, "bad slice range");
  if (cudaSetDevice(h->device) != cudaSuccess) return afail(GLASMA_ERR_CUDA, "cudaSetDevice");
  return h->precision == GLASMA_FP64
             ? glasma::adj64::run_adjoint(h, dt, nsteps, checkpoint_every, z_begin, z_end, num, den, objective, grad_E,
                                          grad_Jp, grad_Jm, grad_JpStat, grad_JmStat)
             : glasma::adj32::run_adjoint(h, dt, nsteps, checkpoint_every, z_begin, z_end, num, den, objective, grad_E,
                                          grad_Jp, grad_Jm, grad_JpStat, grad_JmStat);
}

const char* glasma_adjoint_last_error(void) { return g_adj_error.c_str(); }

}  // extern "C"
