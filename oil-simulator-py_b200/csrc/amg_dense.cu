// Dense operators of the coarse levels: the inverse of the coarsest matrix.
//
// Reference: researchim-ai/oil-simulator-py src/solver/classical_amg.py
//   _v_cycle :1037-1106 (coarsest solve with DOF 0 pinned :1045-1069).
#include "amg.cuh"
#include <algorithm>
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
  if (CL > 8) {
    static const cudaError_t np =
        cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    IMPES_CUDA(np);
  }
  IMPES_CUDA(cudaLaunchKernelEx(&cfg, kern, n, args));
  count_launch();
}

}  // namespace

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
  else launch_gj<16, 1, 32, 16>(n, args, s);
  IMPES_CHECK_LAUNCH();
}

}  // namespace impes
