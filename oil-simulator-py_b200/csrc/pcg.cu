// Jacobi-preconditioned conjugate gradients, the reference's default pressure
// solver: Simulator._solve_pressure_cg_pytorch (simulation.py:1662-1697) as
// called by _impes_pressure_step (:931-966).
//
// Same iteration as the reference: x0 = 0, z = r / diag(A), p = z; stop when
// sqrt(r . z) < tol (absolute) after the x/r update, or after max_iter steps.
// The whole solve is one cooperative launch: a barrier over the grid follows
// each of the two dot products of an iteration, and every block forms alpha, beta
// and the stopping test from the same partials in the same order.  Dot products
// use a fixed partial count and a fixed reduction order, so runs are bitwise
// repeatable.
#include "common.cuh"

namespace impes {
namespace {

constexpr int TBP = 256;                 // rows of a partial sum
constexpr int kBlocks = 296;             // 2 x 148 SMs: fixed partial count
constexpr int kGrid = kBlocks / 2;       // CTAs of two such groups of threads

struct PcgOut {
  double rs;                             // last r . z
  int iters, converged, nan, timeout;
  unsigned arrived;                      // barrier arrivals, grows by kGrid per barrier
};

// All CTAs of the (cooperative) grid; false when the wait gave up.  The limit is looked
// at every kPollBatch polls: compared at each, a solve of 360 iterations took 1.4 % more.
constexpr int kPollBatch = 1024;
__device__ bool grid_barrier(PcgOut* o, unsigned& target, int polls) {
  __shared__ int s_ok;
  target += kGrid;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&o->arrived, 1u);
    int ok = 0;
    for (int q = 0; q < polls && !ok; q += kPollBatch) {
      for (int u = 0; u < kPollBatch; ++u) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(&o->arrived) : "memory");
        if (v >= target) { ok = 1; break; }
      }
    }
    if (!ok) o->timeout = 1;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}
// Sum over the thread's group (256 threads): a partial per group, in a fixed tree.
__device__ __forceinline__ void group_partial(double v, double* sh, double* part) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (threadIdx.x % TBP == 0) {
    double t = 0.0;
    for (int w = 0; w < TBP / 32; ++w) t += sh[wid + w];
    part[blockIdx.x * 2 + threadIdx.x / TBP] = t;
  }
}
// The sum of all partials, the same bits in every thread of the grid.
__device__ __forceinline__ double all_sum(const double* part, double* sh_t) {
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int q = threadIdx.x; q < kBlocks; q += 32) t += __ldcg(part + q);
    t = warp_sum(t);
    if (threadIdx.x == 0) *sh_t = t;
  }
  __syncthreads();
  return *sh_t;
}

// One solve.  p alternates between two arrays, so that the product can form
// p = z + beta p of a row's neighbours while their owners write theirs: the
// direction update needs no barrier of its own.  ONE: at most one row a thread,
// whose x, r, z, p and diagonal stay in registers.
//
// Bound by the two barriers and the chain row pointer -> column -> z, p through
// L2: 7.5 us an iteration at 35,563 rows, against 37 us with a kernel per
// phase and a host read of r . z per iteration.
template <bool ONE>
__global__ void __launch_bounds__(2 * TBP) k_pcg(int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                                                 const double* __restrict__ val, const double* __restrict__ b,
                                                 double* __restrict__ d, double* __restrict__ x,
                                                 double* __restrict__ r, double* z, double* pa, double* pb,
                                                 double* __restrict__ Ap, double* part, double tol, int max_iter,
                                                 int polls, PcgOut* out) {
  __shared__ double sh[2 * TBP / 32], sh_t;
  unsigned target = 0;
  const long long stride = (long long)kBlocks * TBP;
  const long long first = blockIdx.x * 2ll * TBP + threadIdx.x;
  double xi = 0.0, ri = 0.0, zi = 0.0, di = 1.0, pi = 0.0, ai = 0.0;
  double acc = 0.0;
  for (long long i = first; i < n; i += stride) {
    double dv = 0.0;
    for (int e = rowptr[i]; e < rowptr[i + 1]; ++e)
      if (col[e] == i) dv += val[e];
    const double rv = b[i], zv = rv / dv;
    z[i] = zv;
    if (ONE) {
      di = dv; ri = rv; zi = zv;
    } else {
      d[i] = dv; r[i] = rv; x[i] = 0.0;
    }
    acc += rv * zv;
  }
  group_partial(acc, sh, part);
  if (!grid_barrier(out, target, polls)) return;
  double rs = all_sum(part, &sh_t), beta = 0.0;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  int it = 0, conv = rs < 1e-10, nan = !(rs == rs);   // simulation.py:1680-1681
  while (!conv && !nan && it < max_iter) {
    // p = z + beta p, Ap = A p and the partials of p . Ap
    const double* po = (it & 1) ? pa : pb;
    double* pn = (it & 1) ? pb : pa;
    acc = 0.0;
    for (long long i = first; i < n; i += stride) {
      double sum = 0.0;
      const int e1 = rowptr[i + 1];
      for (int e = rowptr[i]; e < e1; ++e) {
        const int c = col[e];
        const double zc = __ldcg(z + c);
        sum += val[e] * (it ? zc + beta * __ldcg(po + c) : zc);
      }
      const double zv = ONE ? zi : z[i];
      const double pv = it ? zv + beta * (ONE ? pi : po[i]) : zv;
      pn[i] = pv;
      if (ONE) { pi = pv; ai = sum; }
      else Ap[i] = sum;
      acc += pv * sum;
    }
    group_partial(acc, sh, part + kBlocks);
    if (!grid_barrier(out, target, polls)) return;
    const double alpha = rs / all_sum(part + kBlocks, &sh_t);
    // x += alpha p, r -= alpha Ap, z = r / d and the partials of r . z
    acc = 0.0;
    for (long long i = first; i < n; i += stride) {
      if (ONE) {
        xi += alpha * pi;
        ri = ri - alpha * ai;
        zi = ri / di;
        z[i] = zi;
        acc += ri * zi;
      } else {
        x[i] += alpha * pn[i];
        const double rv = r[i] - alpha * Ap[i];
        const double zv = rv / d[i];
        r[i] = rv;
        z[i] = zv;
        acc += rv * zv;
      }
    }
    group_partial(acc, sh, part);
    if (!grid_barrier(out, target, polls)) return;
    const double t = all_sum(part, &sh_t);
    beta = t / rs;
    rs = t;
    ++it;
    nan = !(rs == rs);
    conv = !nan && sqrt(rs) < tol;
  }
  if (ONE)
    for (long long i = first; i < n; i += stride) x[i] = xi;
  if (lead) {
    out->rs = rs;
    out->iters = it;
    out->converged = conv;
    out->nan = nan;
  }
}

}  // namespace

// Solves A x = b (x written); returns the iterations taken and whether the
// stopping test fired.  rs_out: the last r.z.  work: the solve's vectors, grown to
// what this size needs.  polls: how often a wait of the grid's barrier looks before it
// gives up (the default is about a second); every CTA then returns.
void pcg_solve(int n, const int* rowptr, const int* col, const double* val, const double* b,
               double* x, double tol, int max_iter, int& iters, bool& converged, double& rs_out,
               DBuf<double>& work, cudaStream_t s, int polls) {
  IMPES_REQUIRE(n > 0 && max_iter >= 0, IMPES_ERR_ARG, "pcg: bad size or iteration limit");
  const bool one = n <= kBlocks * TBP;
  const size_t nv = (size_t)n;
  // z, two directions, and unless they stay in registers d, r and Ap
  work.ensure(nv * (one ? 3 : 6) + 2 * kBlocks + (sizeof(PcgOut) + 7) / 8);
  double* part = work.p;
  PcgOut* out = reinterpret_cast<PcgOut*>(part + 2 * kBlocks);
  double* z = part + 2 * kBlocks + (sizeof(PcgOut) + 7) / 8;
  double *pa = z + nv, *pb = pa + nv;
  double *d = one ? nullptr : pb + nv, *r = one ? nullptr : d + nv, *Ap = one ? nullptr : r + nv;
  IMPES_CUDA(cudaMemsetAsync(out, 0, sizeof(PcgOut), s));
  void* args[] = {&n, &rowptr, &col, &val, &b, &d, &x, &r, &z, &pa, &pb, &Ap, &part, &tol, &max_iter, &polls, &out};
  IMPES_CUDA(cudaLaunchCooperativeKernel(one ? (const void*)k_pcg<true> : (const void*)k_pcg<false>, dim3(kGrid),
                                         dim3(2 * TBP), args, 0, s));
  ::impes::count_launch();
  PcgOut h{};
  IMPES_CUDA(cudaMemcpyAsync(&h, out, sizeof(PcgOut), cudaMemcpyDeviceToHost, s));
  IMPES_CUDA(cudaStreamSynchronize(s));
  iters = h.iters;
  converged = h.converged != 0;
  rs_out = h.rs;
  if (h.timeout) throw Error(IMPES_ERR_TIMEOUT, "pcg: a wait of the grid's barrier ran out");
  if (h.nan)
    throw Error(IMPES_ERR_NAN, h.iters ? "pcg: NaN residual" : "pcg: non-finite right-hand side or diagonal");
}

}  // namespace impes
