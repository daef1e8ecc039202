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
// order.  Measured (B200, both matrices): 32 / 64 / 96 rows 18 / 54 / 121 us, 110
// rows 922 -> 226 us and 124 rows 1169 -> 251 us against a one-CTA elimination in
// shared memory with four barriers a step; in clusters, 200 / 256 rows 486 / 627 us
// (2.4 us a step), 300 / 500 rows 1.33 / 2.33 ms (4.5 us), a matrix in global memory
// having taken 28 ms at 431 rows.
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
// have; IMPES_COARSE_CLUSTER=8 asks for the narrow form (read at setup).  That one
// holds 32 doubles a thread, most of them in local memory: 9.5 / 15.9 ms at 300 / 500
// rows.
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
  // one CTA while 128 columns fit its registers (16 doubles a thread: 2.0 us a pivot
  // step), then 32 columns a CTA in a cluster of 8 (2.4 us) or 16 (4.5 us)
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

enum DnMode { DN_AX = 0, DN_RESID = 1, DN_SWEEP = 2, DN_ADD = 3, DN_PLUS = 4 };

// Epilogue of a product acc = (A X)(i, c):
//  DN_AX: acc;  DN_RESID: I - acc;  DN_SWEEP: x + w (I - acc);  DN_ADD: y + acc;
//  DN_PLUS: x + acc
// The kernels of a forming are one chain of programmatic launches (pdl_fence behind
// it), so matrices that an earlier one writes carry no __restrict__.
template <int MODE>
__device__ __forceinline__ double dn_out(double acc, int i, int c, double w, const double* X, const double* Y,
                                         size_t at) {
  if (MODE == DN_RESID) return (i == c ? 1.0 : 0.0) - acc;
  if (MODE == DN_SWEEP) return X[at] + w * ((i == c ? 1.0 : 0.0) - acc);
  if (MODE == DN_ADD) return Y[at] + acc;
  if (MODE == DN_PLUS) return X[at] + acc;
  return acc;
}

// Y = epilogue(A X) for a CSR matrix A of `rows` rows and a dense X of n
// columns (row-major, leading dimension ld): a warp takes 64 columns, two a lane,
// so every gathered row of X is a contiguous segment.  32 entries of the row are
// loaded at once and handed round by shuffles.  With W = 4 a block's warps share
// one row and 64 columns, warp w taking entries w, w + 4, .. (their sums are
// added in that order): rows of A and R are chains of loads, and some of a capped
// hierarchy's hold half of the columns (748 rows of 25 entries on average, the
// longest 406, and the 184 below them: 34 us a product with W = 1, 17 with W = 4).
// Rows of P are short: W = 1, 256 columns a block (3.6 us, 7.9 with W = 4).
// Bound by L2 (nnz n reads of 8 bytes): used while rows are short.
template <typename TV, int MODE, int W>
__global__ void __launch_bounds__(128) k_dn_spmm(int rows, int n, int ld, const int* __restrict__ rowptr,
                                                 const int* __restrict__ col, const TV* __restrict__ val,
                                                 const TV* __restrict__ inv, const double* X, double* Y) {
  pdl_wait_release();
  constexpr int U = 8;
  __shared__ double2 part[3][32];
  const int i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = ((blockIdx.y * (4 / W) + warp / W) * 32 + lane) * 2;
  const double* Xc = X + min(c, ld - 2);              // (lanes past the last column load, and store nothing)
  const int e0 = rowptr[i] + warp % W, e1 = rowptr[i + 1];
  double a0 = 0.0, a1 = 0.0;
  for (int b = e0; b < e1; b += 32 * W) {             // 32 entries of this warp, one a lane
    const int e = b + W * lane, have = min(32, (e1 - b + W - 1) / W);
    const double v = e < e1 ? (double)val[e] : 0.0;
    const int k = e < e1 ? col[e] : 0;
    for (int q = 0; q < have; q += U) {
      double2 x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kq = __shfl_sync(0xffffffffu, k, q + u);
        x[u] = q + u < have ? *reinterpret_cast<const double2*>(Xc + (size_t)kq * ld) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double vq = __shfl_sync(0xffffffffu, v, q + u);
        a0 += vq * x[u].x;
        a1 += vq * x[u].y;
      }
    }
  }
  if (W > 1) {
    if (warp > 0) part[warp - 1][lane] = make_double2(a0, a1);
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      a0 += part[w][lane].x;
      a1 += part[w][lane].y;
    }
  }
  if (c >= n) return;
  const size_t at = (size_t)i * ld + c;
  const double w = MODE == DN_SWEEP ? (double)(TV(kOmega) * inv[i]) : 0.0;
  double2 r;
  r.x = dn_out<MODE>(a0, i, c, w, X, Y, at);
  r.y = dn_out<MODE>(a1, i, c + 1, w, X, Y, at + 1);
  *reinterpret_cast<double2*>(Y + at) = r;
}

// Y = epilogue(A B), A M x K, B K x N, all row-major with leading dimension ld
// (a multiple of 8), by FP64 matrix instructions (m8n8k4): 32 x 32 tiles of four
// warps (2 x 2), 16-deep slices of A and B through a ring of three buffers
// (cp.async), fragments read from rows padded by four doubles, which keeps the 16
// lanes of a half warp on distinct banks.  Elements outside the matrices are taken
// as zero, whatever the padding columns hold.  DN_SWEEP and DN_PLUS read their x
// from B (X = B there); w = kOmega inv.
// Bound by the FP64 pipe, and by whole tiles an SM: n = 638 24.7 us (21 TFLOP/s),
// 771 47 us, 876 62 us; 64 x 64 tiles with four by four elements a thread took 61,
// 128 and 139 us, bound by shared-memory reads, and 64 x 32 tiles of this kernel
// 53 and 59 us at 771 and 876.
constexpr int kGemmTile = 32, kGemmK = 16, kGemmStages = 3;
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
template <typename TV, int MODE>
__global__ void __launch_bounds__(128) k_dn_gemm(int M, int N, int K, int ld, const double* A, const double* B,
                                                 const TV* __restrict__ inv, double* Y) {
  pdl_wait_release();
  constexpr int BM = kGemmTile, BN = kGemmTile, BK = kGemmK, ST = kGemmStages, LA = BK + 4, LB = BN + 4;
  constexpr int MT = BM / 16, NT = BN / 16;         // 8 x 8 tiles of a warp
  __shared__ __align__(16) double As[ST][BM][LA];
  __shared__ __align__(16) double Bs[ST][BK][LB];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  auto fetch = [&](int st, int k0) {
#pragma unroll
    for (int q = t; q < BM * BK / 2; q += 128) {
      const int r = q / (BK / 2), k = (q % (BK / 2)) * 2;
      const int have = m0 + r < M ? min(2, max(0, K - (k0 + k))) : 0;
      cp_async16(&As[st][r][k], have ? A + (size_t)(m0 + r) * ld + k0 + k : A, 8 * have);
    }
#pragma unroll
    for (int q = t; q < BK * BN / 2; q += 128) {
      const int k = q / (BN / 2), c = (q % (BN / 2)) * 2;
      const int have = k0 + k < K ? min(2, max(0, N - (n0 + c))) : 0;
      cp_async16(&Bs[st][k][c], have ? B + (size_t)(k0 + k) * ld + n0 + c : B, 8 * have);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double acc[MT][NT][2] = {};
  const int steps = (K + BK - 1) / BK;
#pragma unroll
  for (int q = 0; q < ST - 1; ++q) fetch(q, q * BK);    // (past the end: zeros)
  const int wm = (warp >> 1) * (BM / 2) + (lane >> 2), wn = (warp & 1) * (BN / 2) + (lane >> 2), kl = lane & 3;
  for (int q = 0; q < steps; ++q) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");
    __syncthreads();             // slice q is there, and everyone is done with the buffer filled next
    fetch((q + ST - 1) % ST, (q + ST - 1) * BK);
    const int st = q % ST;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      double a[MT], b[NT];
#pragma unroll
      for (int u = 0; u < MT; ++u) a[u] = As[st][wm + 8 * u][k + kl];
#pragma unroll
      for (int v = 0; v < NT; ++v) b[v] = Bs[st][k + kl][wn + 8 * v];
#pragma unroll
      for (int u = 0; u < MT; ++u)
#pragma unroll
        for (int v = 0; v < NT; ++v) mma_f64(acc[u][v][0], acc[u][v][1], a[u], b[v]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int u = 0; u < MT; ++u) {
    const int i = m0 + wm + 8 * u;
    if (i >= M) continue;
    const double w = MODE == DN_SWEEP ? (double)(TV(kOmega) * inv[i]) : 0.0;
#pragma unroll
    for (int v = 0; v < NT; ++v)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int c = n0 + (warp & 1) * (BN / 2) + 8 * v + 2 * kl + x;
        if (c >= N) continue;
        const size_t at = (size_t)i * ld + c;
        Y[at] = dn_out<MODE>(acc[u][v][x], i, c, w, B, Y, at);
      }
  }
}

// What follows from A alone, one warp per row (each output may be null): X1 = W =
// diag(kOmega inv), the first sweep from zero of every column; X2 = W + W (I - A W),
// the second; R = I - A W, the residual after the first.
template <typename TV>
__global__ void __launch_bounds__(256) k_dn_first(int n, int ld, const int* __restrict__ rowptr,
                                                  const int* __restrict__ col, const TV* __restrict__ val,
                                                  const TV* __restrict__ inv, double* X1, double* X2, double* R) {
  pdl_wait_release();
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    const size_t at = (size_t)i * ld;
    const double w = (double)(TV(kOmega) * inv[i]);
    for (int j = lane; j < ld; j += 32) {             // (where A holds no entry, A W is 0)
      const double d = i == j ? 1.0 : 0.0;
      if (X1) X1[at + j] = d * w;
      if (X2) X2[at + j] = d * w + w * d;
      if (R) R[at + j] = d;
    }
    __syncwarp();
    for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
      const int c = col[e];
      const double r = (i == c ? 1.0 : 0.0) - (double)val[e] * (double)(TV(kOmega) * inv[c]);
      if (X2) X2[at + c] = (i == c ? w : 0.0) + w * r;
      if (R) R[at + c] = r;
    }
  }
}
// dense copy of a CSR matrix, one warp per row
template <typename TV>
__global__ void __launch_bounds__(256) k_dn_copy(int n, int ld, const int* __restrict__ rowptr,
                                                 const int* __restrict__ col, const TV* __restrict__ val,
                                                 double* __restrict__ M) {
  pdl_wait_release();
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
  pdl_wait_release();
  const bool use_free = krylov && *free_singular == 0;
  const double* A = use_free ? Afree : Apin;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    E[q] = (c < n && (use_free || c > 0)) ? A[(size_t)i * n + c] : 0.0;
  }
}
// sum = a + b, one = I + a + b
__global__ void k_dn_terms(int n, int ld, const double* a, const double* b, double* sum, double* one) {
  pdl_wait_release();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    const double t = a[q] + b[q];
    sum[q] = t;
    one[q] = (i == c ? 1.0 : 0.0) + t;
  }
}
// E = diag(kOmega inv) T with column 0 (the pinned right-hand side) zero
template <typename TV>
__global__ void k_dn_scale_pin(int n, int ld, const TV* __restrict__ inv, const double* T, double* E) {
  pdl_wait_release();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)n * ld; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q / ld), c = (int)(q % ld);
    E[q] = (c > 0 && c < n) ? (double)(TV(kOmega) * inv[i]) * T[q] : 0.0;
  }
}

// the finished operator, its padding columns zero
__global__ void k_dn_store(int n, int ld, const double* E, double* op) {
  pdl_wait_release();
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
  // an elementwise kernel over n rows
  template <typename... P, typename... A>
  void each(void (*kernel)(int, int, P...), int n, A... args) const {
    launch_pdl(kernel, grid_for((size_t)n * ld, 256, 4), 256, 0, s, n, ld, args...);
    IMPES_CHECK_LAUNCH();
  }
  template <typename TV>
  void first(const Level& L, double* X1, double* X2, double* R) const {
    launch_pdl(k_dn_first<TV>, (unsigned)((L.n + 7) / 8), 256, 0, s, L.n, ld, (const int*)L.rowptr.p,
               (const int*)L.col.p, DV<TV>::val(L), DV<TV>::inv(L), X1, X2, R);
    IMPES_CHECK_LAUNCH();
  }
  template <int MODE, typename TV = double>
  void gemm(int M, int N, int K, const double* A, const double* B, double* Y, const TV* inv = nullptr) const {
    launch_pdl(k_dn_gemm<TV, MODE>, dim3((N + kGemmTile - 1) / kGemmTile, (M + kGemmTile - 1) / kGemmTile), 128, 0, s,
               M, N, K, ld, A, B, inv, Y);
    IMPES_CHECK_LAUNCH();
  }
  template <int MODE, typename TV, int W = 4>
  void spmm(int rows, int n, const int* rp, const int* ci, const TV* v, const TV* inv, const double* X,
            double* Y) const {
    launch_pdl(k_dn_spmm<TV, MODE, W>, dim3(rows, (n + 256 / W - 1) / (256 / W)), 128, 0, s, rows, n, ld, rp, ci, v, inv,
               X, Y);
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

// Forms h.dense_op[slot][dense_mode(krylov)] from the current values of the levels below and at
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
  double* op = h.dense_op[DV<TV>::slot][h.dense_mode(krylov != 0)].p;
  // the coarsest level's operator, in w[0]
  {
    const Level& C = *h.levels.back();
    const int n = C.n;
    if (n <= 500) {
      d.each(k_dn_inverse, n, (const double*)C.lu.p, (const double*)C.lu_free.p, (const int*)(h.iflag.p + 3), krylov,
             w[0]);
    } else {
      // fifty sweeps from zero: W (I + H + ... + H^49), H = I - A W, in nine
      // products as (I + H) s(H^2) s(H^10), s(X) = I + X + X^2 + X^3 + X^4
      double *H = w[1], *P = w[2], *Q = w[3], *S = w[4], *T = w[5], *Z = w[0];
      auto five = [&](const double* X, const double* X2, double* sum, double* out) {
        d.each(k_dn_terms, n, X, X2, sum, out);
        d.gemm<DN_ADD>(n, n, n, X2, sum, out);                // I + X + X^2 + X^2 (X + X^2)
      };
      d.first<TV>(C, nullptr, nullptr, H);
      d.gemm<DN_AX>(n, n, n, H, H, P);                        // H^2
      d.gemm<DN_AX>(n, n, n, P, P, Q);                        // H^4
      five(P, Q, T, S);
      d.gemm<DN_AX>(n, n, n, Q, Q, T);                        // H^8
      d.gemm<DN_AX>(n, n, n, T, P, Z);                        // H^10
      d.gemm<DN_AX>(n, n, n, Z, Z, P);                        // H^20
      five(Z, P, T, Q);
      d.gemm<DN_AX>(n, n, n, S, Q, T);
      d.gemm<DN_PLUS>(n, n, n, H, T, P);
      d.each(k_dn_scale_pin<TV>, n, DV<TV>::inv(C), (const double*)P, Z);
    }
  }
  // each level above it: sweeps on the identity, coarse correction, sweeps
  for (int l = (int)h.levels.size() - 2; l >= dl; --l) {
    const Level& L = *h.levels[l];
    const int n = L.n, nc = L.nc;
    const bool light = n <= h.prm.light_sweep_rows;
    double *E = w[0], *X = w[1], *Y = w[2], *C = w[3], *F = w[4], *A = nullptr;
    if (dense_products(L)) {
      A = w[5];
      launch_pdl(k_dn_copy<TV>, (unsigned)((n + 7) / 8), 256, 0, s, n, ld, (const int*)L.rowptr.p,
                 (const int*)L.col.p, DV<TV>::val(L), A);
      IMPES_CHECK_LAUNCH();
    }
    if (light) {
      d.first<TV>(L, X, nullptr, Y);
    } else {
      d.first<TV>(L, nullptr, Y, nullptr);
      d.product<DN_SWEEP, TV>(L, A, Y, X);
      d.product<DN_RESID, TV>(L, A, X, Y);
    }
    d.spmm<DN_AX, TV>(nc, n, L.rrow.p, L.rcol.p, DV<TV>::rval(L), nullptr, Y, C);
    d.gemm<DN_AX>(nc, n, nc, E, C, F);
    d.spmm<DN_ADD, TV, 1>(n, n, L.prow.p, L.pcol.p, DV<TV>::pval(L), nullptr, F, X);
    for (int q = 0; q < (light ? 1 : 2); ++q) {
      d.product<DN_SWEEP, TV>(L, A, X, Y);
      std::swap(X, Y);
    }
    std::swap(w[0], X == w[1] ? w[1] : w[2]);     // this level's operator is the next one's E
  }
  d.each(k_dn_store, Ld.n, (const double*)w[0], op);
  pdl_fence(s);
}

}  // namespace

// Levels dense_level and below become one operator: from the coarsest level up,
// while a level has at most kDenseRows rows and its products with A on the identity
// stay below kDenseFlops.  A coarsest level of more than 500 rows is taken up to
// kDenseRows whatever its nine products cost (18 n^3: 4.7 GFLOP at 638 rows, 28 at
// 1,152): it saves fifty sweeps a V-cycle.  Forming pays from the break-even number
// of V-cycles after an update on (a solve takes ten to a hundred).  Measured, B200,
// fp64: the operator's rows, time to form it, V-cycle level by level and with it:
//   64x64x1 two-phase, 667:     179 us,  72 ->  38 us, break-even  5
//   47x39x9 two-phase, 523:     318 us, 124 ->  77 us,  7
//   64x64x8 two-phase, 565:     404 us, 153 -> 104 us,  8
//   120x110x25 gas, capped, 748: 195 us, 316 -> 287 us, 7; light sweeps 109 us, 8
//   coarsest of 638 rows, 459 a row:  330 us, 623 -> 489 us, 2.5
//   coarsest of 947 rows, 544 a row:  756 us, 509 -> 379 us, 6
//   coarsest of 771 / 1,035 / 1,113 rows, 14 a row: 508 / 902 / 1,072 us, 130 -> 26 us,
//     5 / 9 / 11, so past kDenseRows a solve of ten V-cycles would lose
// One to three V-cycles after each update cost up to that forming more than level by
// level, on these sizes 0.1 to 1 ms.
//
// Six work matrices and the operators stay with the handle (7 to 10 n^2 doubles: 33 MB at
// 771 rows, up to 106 MB at 1,152), since every update forms them again, from graphs too.
// A program with many small hierarchies would run out of device memory by them, so
// they are taken only while they are at most 1/kDenseShare of what is free; the
// levels' own kernels serve otherwise.
constexpr size_t kDenseShare = 64;
constexpr int kDenseRows = 1152;
constexpr double kDenseFlops = 4e9;
void amg_dense_setup(AMG& h) {
  h.dense_level = -1;
  h.dense_invalidate();
  auto release = [&] {
    h.dense_work.release();
    for (auto& a : h.dense_op) for (auto& b : a) b.release();
  };
  release();                                 // (of the hierarchy before)
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
  const int ld = (D.n + 7) / 8 * 8;
  const size_t sz = (size_t)D.n * ld;
  const int modes = C.n > 500 ? 1 : 2, slots = h.prm.mixed_precision ? 2 : 1;
  size_t free_b = 0, total_b = 0;
  IMPES_CUDA(cudaMemGetInfo(&free_b, &total_b));
  if ((6 + (size_t)modes * slots) * sz * sizeof(double) > free_b / kDenseShare) return;
  try {
    h.dense_work.alloc(6 * sz);
    for (int q = 0; q < slots; ++q)
      for (int k = 0; k < modes; ++k) h.dense_op[q][k].alloc(sz);
  } catch (const Error&) {                   // taken by someone else since
    cudaGetLastError();
    release();
    return;
  }
  h.dense_modes = modes;
  h.dense_ld = ld;
  h.dense_level = dl;
}

void amg_dense_form(AMG& h, int slot, bool krylov, cudaStream_t s) {
  if (h.dense_level < 0) return;
  if (slot == 0) dense_form<double>(h, krylov ? 1 : 0, s);
  else dense_form<float>(h, krylov ? 1 : 0, s);
  if (!stream_capturing(s)) h.dense_valid[slot][h.dense_mode(krylov)] = true;
}

template <typename T>
void dense_apply(const AMG& h, bool krylov, const T* b, T* x, cudaStream_t s) {
  const int n = h.levels[h.dense_level]->n;
  launch_pdl(k_dn_apply<T>, (n + 3) / 4, 128, h.dense_ld * sizeof(double), s, n, h.dense_ld,
             (const double*)h.dense_op[sizeof(T) == 4][h.dense_mode(krylov)].p, b, x);
  IMPES_CHECK_LAUNCH();
}
template void dense_apply<double>(const AMG&, bool, const double*, double*, cudaStream_t);
template void dense_apply<float>(const AMG&, bool, const float*, float*, cudaStream_t);

}  // namespace impes
