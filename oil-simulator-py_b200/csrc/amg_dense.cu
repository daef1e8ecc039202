// Dense operators of the coarse levels: the inverse of the coarsest matrix, and
// the V-cycle of the coarse levels as one matrix.
//
// Reference: researchim-ai/oil-simulator-py src/solver/classical_amg.py
//   _v_cycle :1037-1106 (coarsest solve with DOF 0 pinned :1045-1069).
#include "amg.cuh"
#include <algorithm>
#include <cstdlib>
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace impes {
namespace {

// Dense copies of the coarsest matrix, one warp per row: Mpin with row and
// column 0 replaced by e_0 (classical_amg.py:1051-1055), Mfree as it is.
template <typename TV>
__global__ void __launch_bounds__(256) k_dense_pair(int n, const int* __restrict__ rowptr,
                                                    const int* __restrict__ col, const TV* __restrict__ val,
                                                    double* __restrict__ Mpin, double* __restrict__ Mfree) {
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    double* a = Mpin + (size_t)i * n;
    double* f = Mfree + (size_t)i * n;
    for (int j = lane; j < n; j += 32) {
      a[j] = (i == 0 && j == 0) ? 1.0 : 0.0;
      f[j] = 0.0;
    }
    __syncwarp();
    for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
      const int j = col[e];
      const double v = (double)val[e];
      f[j] = v;
      if (i != 0 && j != 0) a[j] = v;
    }
  }
}

// ------------------------------------------------ Gauss-Jordan inversion
// In-place inverse with partial pivoting (largest |value| of the column, ties to
// the lower row), the matrix held in registers for the whole elimination: lane
// and column block give a thread's column j, its row group rg the rows
// rg RPT .. rg RPT + RPT - 1.  A cluster of CL CTAs shares one matrix, CTA c
// holding columns [32 CB c, 32 CB (c + 1)); cluster b inverts args.M[b] (the
// pinned and the unpinned matrix in one launch).
//
// A pivot step is a dependent chain, so its length bounds the kernel, not bytes:
// column k (all rows) goes to every CTA's shared memory; every warp finds the
// pivot itself (integer maxima of the value's bits, so no block reduction); the
// threads of rows k and p publish their elements of those rows; then every
// element is updated in its register with one shared-memory read and one fused
// multiply-add (the two rows that change places are set afterwards by the warps
// that hold them), and the owner of column k + 1 publishes it.  Two block
// barriers a step (one of them the cluster's when CL > 1).  Each element gets
// the operations of the textbook in-place elimination with row swaps, in that
// order.  Measured (B200, both matrices): 110 rows 922 -> 226 us, 124 rows 1169
// -> 252 us against a one-CTA elimination in shared memory with four barriers a
// step; about 200 rows 1462 -> 404 us against one in global memory.
struct GJArgs {
  double* M[2];
  int* singular[2];
};
constexpr int kGJMax = 512;
template <int CL, int CB, int RG, int RPT>
__global__ void __launch_bounds__(32 * CB * RG) k_gauss_jordan(int n, GJArgs args) {
  static_assert(RPT % 2 == 0, "rows are read in pairs");
  constexpr int NR = RG * RPT;                 // rows held
  __shared__ __align__(16) double s_col[2][NR];     // column k of the current matrix
  __shared__ double s_rp[32 * CB], s_rk[32 * CB];   // this CTA's part of rows p and k
  __shared__ double s_inv;
  __shared__ int s_perm[kGJMax];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cb = warp % CB, rg = warp / CB;
  const int which = blockIdx.x / CL, rank = blockIdx.x % CL;
  const int jl = cb * 32 + lane, j = rank * 32 * CB + jl;
  double* G = args.M[which];
  double a[RPT];
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    const int i = rg * RPT + u;
    a[u] = (i < n && j < n) ? G[(size_t)i * n + j] : 0.0;
  }
  // column 0, to every CTA of the cluster
  for (int i = threadIdx.x; i < NR; i += blockDim.x) s_col[0][i] = i < n ? G[(size_t)i * n] : 0.0;
  bool singular = false;
  for (int k = 0; k < n; ++k) {
    const double* col = s_col[k & 1];
    double* ncol = s_col[(k + 1) & 1];
    // (the first one also: every CTA has to be running before another writes to it)
    if (CL > 1) cg::this_cluster().sync();
    else __syncthreads();
    // the pivot: key 0 for rows outside [k, n) and NaN, else the bits of |v| + 1
    unsigned long long best = 0;
    int bi = k;
#pragma unroll
    for (int q = 0; q < (NR + 31) / 32; ++q) {
      const int i = lane + 32 * q;
      if (i >= k && i < n) {
        const double v = fabs(col[i]);
        const unsigned long long key = v >= 0.0 ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
        if (key > best) { best = key; bi = i; }
      }
    }
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
    const bool top = (unsigned)(best >> 32) == hi;
    const unsigned lo = __reduce_max_sync(0xffffffffu, top ? (unsigned)best : 0u);
    const bool mine = top && (unsigned)best == lo;
    const int p = (hi | lo) ? (int)__reduce_min_sync(0xffffffffu, mine ? (unsigned)bi : 0xffffffffu) : k;
    if (threadIdx.x == 0) {
      const double piv = col[p];
      if (!(fabs(piv) > 0.0)) singular = true;
      s_inv = piv != 0.0 ? 1.0 / piv : 0.0;
      s_perm[k] = p;
    }
    // rows p and k of this CTA's columns
    if (rg == p / RPT) {
#pragma unroll
      for (int u = 0; u < RPT; ++u) if (rg * RPT + u == p) s_rp[jl] = a[u];
    }
    if (rg == k / RPT) {
#pragma unroll
      for (int u = 0; u < RPT; ++u) if (rg * RPT + u == k) s_rk[jl] = a[u];
    }
    __syncthreads();
    const double inv = s_inv;
    const double sr = (j == k) ? inv : s_rp[jl] * inv;
    // column k: 0 - f sr
    if (j == k)
#pragma unroll
      for (int u = 0; u < RPT; ++u) a[u] = 0.0;
#pragma unroll
    for (int u = 0; u < RPT; u += 2) {
      const double2 f = *reinterpret_cast<const double2*>(col + rg * RPT + u);
      a[u] = a[u] - f.x * sr;
      a[u + 1] = a[u + 1] - f.y * sr;
    }
    if (rg == p / RPT) {              // row p: the old row k
      const double v = ((j == k) ? 0.0 : s_rk[jl]) - col[k] * sr;
#pragma unroll
      for (int u = 0; u < RPT; ++u) a[u] = (rg * RPT + u == p) ? v : a[u];
    }
    if (rg == k / RPT) {              // row k: the scaled pivot row
#pragma unroll
      for (int u = 0; u < RPT; ++u) a[u] = (rg * RPT + u == k) ? sr : a[u];
    }
    if (k + 1 < n && rank == (k + 1) / (32 * CB)) {
      if (j == k + 1)
#pragma unroll
        for (int u = 0; u < RPT; ++u) ncol[rg * RPT + u] = a[u];
      if (CL > 1) {
        __syncthreads();
        cg::cluster_group cl = cg::this_cluster();
        for (int t = threadIdx.x; t < (CL - 1) * NR; t += blockDim.x) {
          const int i = t % NR;
          const int c = (rank + 1 + t / NR) % CL;
          cl.map_shared_rank(ncol, c)[i] = ncol[i];
        }
      }
    }
  }
  __syncthreads();
  // row interchanges are undone as column interchanges, last first: s_pos[c] is
  // the final place of column c
  __shared__ int s_at[kGJMax], s_pos[kGJMax];
  for (int c = threadIdx.x; c < n; c += blockDim.x) s_at[c] = c;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = n - 1; k >= 0; --k) {
      const int p = s_perm[k];
      if (p != k) { const int t = s_at[k]; s_at[k] = s_at[p]; s_at[p] = t; }
    }
  __syncthreads();
  for (int c = threadIdx.x; c < n; c += blockDim.x) s_pos[s_at[c]] = c;
  __syncthreads();
  if (j < n) {
    const int jp = s_pos[j];
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      const int i = rg * RPT + u;
      if (i < n) G[(size_t)i * n + jp] = a[u];
    }
  }
  if (singular && rank == 0) *args.singular[which] = 1;   // thread 0
  // no CTA leaves while another may still write to its shared memory
  if (CL > 1) cg::this_cluster().sync();
}

template <int CL, int CB, int RG, int RPT>
void launch_gj(int n, const GJArgs& args, cudaStream_t s) {
  auto* kern = k_gauss_jordan<CL, CB, RG, RPT>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * CL);
  cfg.blockDim = dim3(32 * CB * RG);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CL > 1 ? 1 : 0;
  if (CL > 8) allow_wide_cluster((const void*)kern);
  IMPES_CUDA(cudaLaunchKernelEx(&cfg, kern, n, args));
  count_launch();
}

}  // namespace

// Sixteen CTAs need that many free SMs in one GPC, which a part of a GPU may not
// have; IMPES_COARSE_CLUSTER=8 asks for the narrow form (read at setup).
int coarse_cluster_size() {
  const char* ev = getenv("IMPES_COARSE_CLUSTER");
  if (ev && atoi(ev) == 8) return 8;
  auto* kern = k_gauss_jordan<16, 1, 32, 16>;
  allow_wide_cluster((const void*)kern);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * 16);
  cfg.blockDim = dim3(1024);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters >= 1) return 16;
  cudaGetLastError();
  return 8;
}

void coarse_factor(AMG& h, Level& L, cudaStream_t s, bool from_fp32) {
  if (L.n > 500 || L.n == 0) return;
  const int n = L.n;
  // the reference's pinned matrix (row/column 0 replaced by e_0) and the
  // unpinned one used inside FGMRES (the pinned solve would freeze x[0] there)
  L.lu.ensure((size_t)n * n);
  L.lu_free.ensure((size_t)n * n);
  const unsigned grid = (unsigned)((n + 7) / 8);
  if (from_fp32)
    k_dense_pair<float><<<grid, 256, 0, s>>>(n, L.rowptr.p, L.col.p, L.valf.p, L.lu.p, L.lu_free.p);
  else
    k_dense_pair<double><<<grid, 256, 0, s>>>(n, L.rowptr.p, L.col.p, L.val.p, L.lu.p, L.lu_free.p);
  ::impes::count_launch();
  IMPES_CHECK_LAUNCH();
  IMPES_CUDA(cudaMemsetAsync(h.iflag.p + 2, 0, 2 * sizeof(int), s));
  const GJArgs args{{L.lu.p, L.lu_free.p}, {h.iflag.p + 2, h.iflag.p + 3}};
  // one CTA while 128 columns fit its registers (16 doubles a thread), then 32
  // columns a CTA in a cluster of 8 or 16 (2.1 us a pivot step in one CTA, about
  // as much in a cluster of 8)
  if (n <= 32) launch_gj<1, 1, 8, 4>(n, args, s);
  else if (n <= 64) launch_gj<1, 2, 8, 8>(n, args, s);
  else if (n <= 96) launch_gj<1, 3, 8, 12>(n, args, s);
  else if (n <= 128) launch_gj<1, 4, 8, 16>(n, args, s);
  else if (n <= 256) launch_gj<8, 1, 32, 8>(n, args, s);
  else if (h.coarse_cluster == 16) launch_gj<16, 1, 32, 16>(n, args, s);
  else launch_gj<8, 2, 16, 32>(n, args, s);
  IMPES_CHECK_LAUNCH();
}

namespace {
// ---------------------------------------------- one operator for a coarse V-cycle
// A V-cycle from zero is a linear map of its right-hand side, fixed while the
// matrix values are: below Level h.dense_level it is applied as ONE dense
// product instead of up to seven dependent kernels a level (and fifty sweeps on
// a coarsest level of more than 500 rows).  The operator is formed after every
// change of values by running the same sweeps, residuals and transfers on the
// identity (all columns at once), coarsest level first.
//
// Always float64, also for the fp32 V-cycle (whose level values it is formed
// from): it holds the coarsest inverse, which stays float64 there too.
constexpr double kOmega = 0.7;  // classical_amg.py:1022

enum DnMode { DN_AX = 0, DN_RESID = 1, DN_SWEEP = 2, DN_ADD = 3 };

// Epilogue of a product acc = (A X)(i, c):
//  DN_AX: acc;  DN_RESID: I - acc;  DN_SWEEP: x + w (I - acc);  DN_ADD: y + acc
template <int MODE>
__device__ __forceinline__ double dn_out(double acc, int i, int c, double w, const double* X, const double* Y,
                                         size_t at) {
  if (MODE == DN_RESID) return (i == c ? 1.0 : 0.0) - acc;
  if (MODE == DN_SWEEP) return X[at] + w * ((i == c ? 1.0 : 0.0) - acc);
  if (MODE == DN_ADD) return Y[at] + acc;
  return acc;
}

// Y = epilogue(A X) for a CSR matrix A of `rows` rows and a dense X of n
// columns (row-major, leading dimension ld): a block takes one row of A and 256
// columns, two a thread, so every gathered row of X is one contiguous segment.
// Bound by L2 (nnz n reads of 8 bytes): used while rows are short.
template <typename TV, int MODE>
__global__ void __launch_bounds__(128) k_dn_spmm(int rows, int n, int ld, const int* __restrict__ rowptr,
                                                 const int* __restrict__ col, const TV* __restrict__ val,
                                                 const TV* __restrict__ inv, const double* __restrict__ X,
                                                 double* Y) {
  const int i = blockIdx.x;
  const int c = (blockIdx.y * 128 + threadIdx.x) * 2;
  if (c >= n) return;
  double a0 = 0.0, a1 = 0.0;
  const int e1 = rowptr[i + 1];
  int e = rowptr[i];
  for (; e + 4 <= e1; e += 4) {
    double2 x[4];
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      v[u] = (double)val[e + u];
      x[u] = *reinterpret_cast<const double2*>(X + (size_t)col[e + u] * ld + c);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) { a0 += v[u] * x[u].x; a1 += v[u] * x[u].y; }
  }
  for (; e < e1; ++e) {
    const double v = (double)val[e];
    const double2 x = *reinterpret_cast<const double2*>(X + (size_t)col[e] * ld + c);
    a0 += v * x.x;
    a1 += v * x.y;
  }
  const size_t at = (size_t)i * ld + c;
  const double w = MODE == DN_SWEEP ? (double)(TV(kOmega) * inv[i]) : 0.0;
  double2 r;
  r.x = dn_out<MODE>(a0, i, c, w, X, Y, at);
  r.y = dn_out<MODE>(a1, i, c + 1, w, X, Y, at + 1);
  *reinterpret_cast<double2*>(Y + at) = r;
}

// Y = epilogue(A B), A M x K, B K x N, all row-major with leading dimension ld
// (a multiple of 8): 64 x 64 tiles, 4 x 4 elements a thread, the next 16-deep
// slice of A and B in registers while the current one is multiplied.  Bound by
// the FP64 pipe.  DN_SWEEP reads its x from B (X = B there); w = kOmega inv.
template <typename TV, int MODE>
__global__ void __launch_bounds__(256) k_dn_gemm(int M, int N, int K, int ld, const double* __restrict__ A,
                                                 const double* __restrict__ B, const TV* __restrict__ inv, double* Y) {
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ __align__(16) double As[2][BK][BM + 2];
  __shared__ __align__(16) double Bs[2][BK][BN];
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  double ra[4], rb[4];
  // A: rows m0 + t / 4 .. , four consecutive k a thread; B: row t / 16, four columns
  auto load = [&](int k0) {
    const int m = m0 + (t >> 2), ka = k0 + (t & 3) * 4;
#pragma unroll
    for (int u = 0; u < 4; ++u) ra[u] = (m < M && ka + u < K) ? A[(size_t)m * ld + ka + u] : 0.0;
    const int kb = k0 + (t >> 4), nb = n0 + (t & 15) * 4;
#pragma unroll
    for (int u = 0; u < 4; ++u) rb[u] = (kb < K && nb + u < N) ? B[(size_t)kb * ld + nb + u] : 0.0;
  };
  auto store = [&](int st) {
#pragma unroll
    for (int u = 0; u < 4; ++u) As[st][(t & 3) * 4 + u][t >> 2] = ra[u];
#pragma unroll
    for (int u = 0; u < 4; ++u) Bs[st][t >> 4][(t & 15) * 4 + u] = rb[u];
  };
  double acc[4][4] = {};
  load(0);
  store(0);
  __syncthreads();
  int st = 0;
  for (int k0 = 0; k0 < K; k0 += BK) {
    const bool more = k0 + BK < K;
    if (more) load(k0 + BK);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      double a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; u += 2) {
        const double2 va = *reinterpret_cast<const double2*>(&As[st][k][ty * 4 + u]);
        a[u] = va.x; a[u + 1] = va.y;
        const double2 vb = *reinterpret_cast<const double2*>(&Bs[st][k][tx * 2 + 16 * u]);
        b[u] = vb.x; b[u + 1] = vb.y;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] += a[u] * b[v];
    }
    if (more) store(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = m0 + ty * 4 + u;
    if (i >= M) continue;
    const double w = MODE == DN_SWEEP ? (double)(TV(kOmega) * inv[i]) : 0.0;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int c = n0 + tx * 2 + 16 * (v & 2) + (v & 1);
      if (c >= N) continue;
      const size_t at = (size_t)i * ld + c;
      Y[at] = dn_out<MODE>(acc[u][v], i, c, w, B, Y, at);
    }
  }
}

// X = diag(kOmega inv) (the first sweep from zero of every column)
template <typename TV>
__global__ void k_dn_diag(int n, int ld, const TV* __restrict__ inv, double* __restrict__ X) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    X[q] = i == c ? (double)(TV(kOmega) * inv[i]) : 0.0;
  }
}
// dense copy of a CSR matrix, one warp per row
template <typename TV>
__global__ void __launch_bounds__(256) k_dn_copy(int n, int ld, const int* __restrict__ rowptr,
                                                 const int* __restrict__ col, const TV* __restrict__ val,
                                                 double* __restrict__ M) {
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    double* m = M + (size_t)i * ld;
    for (int j = lane; j < ld; j += 32) m[j] = 0.0;
    __syncwarp();
    for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) m[col[e]] = (double)val[e];
  }
}
// the coarsest solve's operator: the pinned inverse with b[0] taken as 0, or in
// Krylov mode the unpinned one unless it was singular (k_coarse_apply's choice)
__global__ void k_dn_inverse(int n, int ld, const double* __restrict__ Apin, const double* __restrict__ Afree,
                             const int* __restrict__ free_singular, int krylov, double* __restrict__ E) {
  const bool use_free = krylov && *free_singular == 0;
  const double* A = use_free ? Afree : Apin;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    E[q] = (c < n && (use_free || c > 0)) ? A[(size_t)i * n + c] : 0.0;
  }
}
// out = I + a (+ b)
__global__ void k_dn_one_plus(int n, int ld, const double* __restrict__ a, const double* __restrict__ b,
                              double* __restrict__ out) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    out[q] = (i == c ? 1.0 : 0.0) + (b ? a[q] + b[q] : a[q]);
  }
}
// E = diag(kOmega inv) T with column 0 (the pinned right-hand side) zero
template <typename TV>
__global__ void k_dn_scale_pin(int n, int ld, const TV* __restrict__ inv, const double* __restrict__ T,
                               double* __restrict__ E) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    E[q] = (c > 0 && c < n) ? (double)(TV(kOmega) * inv[i]) * T[q] : 0.0;
  }
}

// the finished operator, its padding columns zero
__global__ void k_dn_store(int n, int ld, const double* __restrict__ E, double* __restrict__ op) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x)
    op[q] = (int)(q % ld) < n ? E[q] : 0.0;
}

// x = Op b, one warp per row, b staged in shared memory.  The first part of the
// row is loaded before the wait on the kernel that writes b: Op was complete
// before that kernel's own predecessors started.
template <typename T>
__global__ void __launch_bounds__(128) k_dn_apply(int n, int ld, const double* __restrict__ Op, const T* b, T* x) {
  extern __shared__ __align__(16) double s_x[];
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
  const double2* row = reinterpret_cast<const double2*>(Op + (size_t)(i < n ? i : 0) * ld);
  const int n2 = ld / 2;
  constexpr int PF = 8;
  double2 pre[PF];
#pragma unroll
  for (int u = 0; u < PF; ++u) pre[u] = lane + 32 * u < n2 ? row[lane + 32 * u] : make_double2(0.0, 0.0);
  pdl_wait_release();
  for (int q = threadIdx.x; q < ld; q += 128) s_x[q] = q < n ? (double)b[q] : 0.0;
  __syncthreads();
  const double2* s2 = reinterpret_cast<const double2*>(s_x);
  double a0 = 0.0, a1 = 0.0;
#pragma unroll
  for (int u = 0; u < PF; ++u)
    if (lane + 32 * u < n2) {
      const double2 s = s2[lane + 32 * u];
      a0 += pre[u].x * s.x;
      a1 += pre[u].y * s.y;
    }
  for (int q = lane + 32 * PF; q < n2; q += 32) {
    const double2 m = row[q], s = s2[q];
    a0 += m.x * s.x;
    a1 += m.y * s.y;
  }
  const double acc = warp_sum(a0 + a1);
  if (lane == 0 && i < n) x[i] = (T)acc;
}

template <typename TV> struct DV;
template <> struct DV<double> {
  static constexpr int slot = 0;
  static const double* val(const Level& L) { return L.val.p; }
  static const double* inv(const Level& L) { return L.inv_relax.p; }
  static const double* pval(const Level& L) { return L.pval.p; }
  static const double* rval(const Level& L) { return L.rval.p; }
};
template <> struct DV<float> {
  static constexpr int slot = 1;
  static const float* val(const Level& L) { return L.valf.p; }
  static const float* inv(const Level& L) { return L.inv_relaxf.p; }
  static const float* pval(const Level& L) { return L.pvalf.p; }
  static const float* rval(const Level& L) { return L.rvalf.p; }
};

struct Dense {
  int ld;
  cudaStream_t s;
  unsigned ew(int n) const { return grid_for((size_t)n * ld, 256, 4); }
  template <int MODE, typename TV = double>
  void gemm(int M, int N, int K, const double* A, const double* B, double* Y, const TV* inv = nullptr) const {
    k_dn_gemm<TV, MODE><<<dim3((N + 63) / 64, (M + 63) / 64), 256, 0, s>>>(M, N, K, ld, A, B, inv, Y);
    count_launch();
    IMPES_CHECK_LAUNCH();
  }
  template <int MODE, typename TV>
  void spmm(int rows, int n, const int* rp, const int* ci, const TV* v, const TV* inv, const double* X,
            double* Y) const {
    k_dn_spmm<TV, MODE><<<dim3(rows, (n + 255) / 256), 128, 0, s>>>(rows, n, ld, rp, ci, v, inv, X, Y);
    count_launch();
    IMPES_CHECK_LAUNCH();
  }
  // Y = epilogue(A X) with the level's A (dense copy Ad when given)
  template <int MODE, typename TV>
  void product(const Level& L, const double* Ad, const double* X, double* Y) const {
    if (Ad) gemm<MODE, TV>(L.n, L.n, L.n, Ad, X, Y, DV<TV>::inv(L));
    else spmm<MODE, TV>(L.n, L.n, L.rowptr.p, L.col.p, DV<TV>::val(L), DV<TV>::inv(L), X, Y);
  }
};

// The level's products run as dense ones: FP64 work n^3 against nnz n gathers
// of 8 bytes from L2.
inline bool dense_products(const Level& L) { return L.avg_row >= L.n / 6; }

// Forms h.dense_op[slot][krylov] from the current values of the levels below and at
// h.dense_level (fp64 ones or the fp32 chain's).
template <typename TV>
void dense_form(AMG& h, int krylov, cudaStream_t s) {
  const int dl = h.dense_level;
  Level& Ld = *h.levels[dl];
  const int ld = h.dense_ld;
  const Dense d{ld, s};
  const size_t sz = (size_t)Ld.n * ld;
  double* w[6];
  for (int q = 0; q < 6; ++q) w[q] = h.dense_work.p + q * sz;
  double* op = h.dense_op[DV<TV>::slot][krylov].p;
  // the coarsest level's operator, in w[0]
  {
    const Level& C = *h.levels.back();
    const int n = C.n;
    if (n <= 500) {
      k_dn_inverse<<<d.ew(n), 256, 0, s>>>(n, ld, C.lu.p, C.lu_free.p, h.iflag.p + 3, krylov, w[0]);
      count_launch();
    } else {
      // fifty sweeps from zero: W (I + H + ... + H^49), H = I - A W, by doubling
      // the number of terms: S_2m = S_m + H^m S_m
      double *H = w[1], *P = w[2], *S = w[3], *Q = w[4], *A = w[5];
      k_dn_diag<TV><<<d.ew(n), 256, 0, s>>>(n, ld, DV<TV>::inv(C), P);
      count_launch();
      if (dense_products(C)) {
        k_dn_copy<TV><<<(unsigned)((n + 7) / 8), 256, 0, s>>>(n, ld, C.rowptr.p, C.col.p, DV<TV>::val(C), A);
        count_launch();
      }
      d.product<DN_RESID, TV>(C, dense_products(C) ? A : nullptr, P, H);            // H
      d.gemm<DN_AX>(n, n, n, H, H, P);                                        // H^2
      k_dn_one_plus<<<d.ew(n), 256, 0, s>>>(n, ld, H, P, S);                  // S_3
      count_launch();
      d.gemm<DN_AX>(n, n, n, P, H, Q);                                        // H^3
      for (int m = 3; m < 24; m *= 2) {
        IMPES_CUDA(cudaMemcpyAsync(P, S, sz * sizeof(double), cudaMemcpyDeviceToDevice, s));
        d.gemm<DN_ADD>(n, n, n, Q, P, S);                                     // S_2m
        d.gemm<DN_AX>(n, n, n, Q, Q, A);                                      // H^2m
        std::swap(Q, A);
      }
      d.gemm<DN_AX>(n, n, n, H, S, P);
      k_dn_one_plus<<<d.ew(n), 256, 0, s>>>(n, ld, P, nullptr, S);            // S_25 = I + H S_24
      count_launch();
      d.gemm<DN_AX>(n, n, n, Q, H, A);                                        // H^25
      IMPES_CUDA(cudaMemcpyAsync(P, S, sz * sizeof(double), cudaMemcpyDeviceToDevice, s));
      d.gemm<DN_ADD>(n, n, n, A, P, S);                                       // S_50
      k_dn_scale_pin<TV><<<d.ew(n), 256, 0, s>>>(n, ld, DV<TV>::inv(C), S, w[0]);
      count_launch();
    }
    IMPES_CHECK_LAUNCH();
  }
  // each level above it: sweeps on the identity, coarse correction, sweeps
  for (int l = (int)h.levels.size() - 2; l >= dl; --l) {
    const Level& L = *h.levels[l];
    const int n = L.n, nc = L.nc;
    const bool light = n <= h.prm.light_sweep_rows;
    double *E = w[0], *X = w[1], *Y = w[2], *C = w[3], *F = w[4], *A = nullptr;
    if (dense_products(L)) {
      A = w[5];
      k_dn_copy<TV><<<(unsigned)((n + 7) / 8), 256, 0, s>>>(n, ld, L.rowptr.p, L.col.p, DV<TV>::val(L), A);
      count_launch();
    }
    k_dn_diag<TV><<<d.ew(n), 256, 0, s>>>(n, ld, DV<TV>::inv(L), X);
    count_launch();
    for (int q = 1; q < (light ? 1 : 3); ++q) {
      d.product<DN_SWEEP, TV>(L, A, X, Y);
      std::swap(X, Y);
    }
    d.product<DN_RESID, TV>(L, A, X, Y);
    d.spmm<DN_AX, TV>(nc, n, L.rrow.p, L.rcol.p, DV<TV>::rval(L), nullptr, Y, C);
    d.gemm<DN_AX>(nc, n, nc, E, C, F);
    d.spmm<DN_ADD, TV>(n, n, L.prow.p, L.pcol.p, DV<TV>::pval(L), nullptr, F, X);
    for (int q = 0; q < (light ? 1 : 2); ++q) {
      d.product<DN_SWEEP, TV>(L, A, X, Y);
      std::swap(X, Y);
    }
    std::swap(w[0], X == w[1] ? w[1] : w[2]);     // this level's operator is the next one's E
  }
  k_dn_store<<<d.ew(Ld.n), 256, 0, s>>>(Ld.n, ld, w[0], op);
  count_launch();
  IMPES_CHECK_LAUNCH();
}

}  // namespace

// Levels dense_level and below become one operator: from the coarsest level up,
// while a level has at most kDenseRows rows and its products on the identity
// stay below kDenseFlops, so that forming it (at about 9 TFLOP/s) pays after
// about ten V-cycles (an update is followed by ten to a hundred of them).  A
// coarsest level of more than 500 rows is taken whatever it costs: it saves
// fifty sweeps a V-cycle.  Measured against the per-level kernels (B200, all
// update costs included): 64x64 two-phase step (663 rows down) 7.18 -> 5.67 ms,
// black-oil 100x100x20 step (coarsest 665 rows) 105.0 -> 73.1 ms, 100 stand-alone
// V-cycles of a 64x64x8 system (565 rows down) 20.1 -> 15.5 ms, mixed 1e6-cell
// step (776 rows down, light sweeps) 72.8 -> 70.6 ms.
constexpr int kDenseRows = 1152;
constexpr double kDenseFlops = 4e9;
void amg_dense_setup(AMG& h) {
  h.dense_level = -1;
  h.dense_invalidate();
  if (h.prm.smoother != IMPES_SMOOTHER_L1_JACOBI || h.tail_level >= 0 || h.stail_level >= 0) return;
  const Level& C = *h.levels.back();
  int dl = (int)h.levels.size() - 1;
  if (dl < 1 || C.n > kDenseRows) return;
  for (; dl > 1; --dl) {
    const Level& L = *h.levels[dl - 1];
    const double terms = dense_products(L) ? (double)L.n * L.n : (double)L.nnz;
    const double products = L.n <= h.prm.light_sweep_rows ? 2.0 : 5.0;
    if (L.n > kDenseRows || 2.0 * products * terms * L.n > kDenseFlops) break;
  }
  const Level& D = *h.levels[dl];
  if (D.coarsest && D.n <= 500) return;      // already one product (k_coarse_apply)
  h.dense_level = dl;
  h.dense_ld = (D.n + 7) / 8 * 8;
  const size_t sz = (size_t)D.n * h.dense_ld;
  h.dense_work.ensure(6 * sz);
  for (int q = 0; q < (h.prm.mixed_precision ? 2 : 1); ++q)
    for (int k = 0; k < 2; ++k) h.dense_op[q][k].ensure(sz);
}

void amg_dense_form(AMG& h, int slot, bool krylov, cudaStream_t s) {
  if (h.dense_level < 0) return;
  if (slot == 0) dense_form<double>(h, krylov ? 1 : 0, s);
  else dense_form<float>(h, krylov ? 1 : 0, s);
  if (!stream_capturing(s)) h.dense_valid[slot][krylov ? 1 : 0] = true;
}

template <typename T>
void dense_apply(const AMG& h, bool krylov, const T* b, T* x, cudaStream_t s) {
  const int n = h.levels[h.dense_level]->n;
  launch_pdl(k_dn_apply<T>, (n + 3) / 4, 128, h.dense_ld * sizeof(double), s, n, h.dense_ld,
             (const double*)h.dense_op[sizeof(T) == 4][krylov ? 1 : 0].p, b, x);
  IMPES_CHECK_LAUNCH();
}
template void dense_apply<double>(const AMG&, bool, const double*, double*, cudaStream_t);
template void dense_apply<float>(const AMG&, bool, const float*, float*, cudaStream_t);

}  // namespace impes
