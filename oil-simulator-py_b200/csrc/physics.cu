// Pressure assembly (K1) and explicit saturation update (K4) of the IMPES step.
//
// Reference: researchim-ai/oil-simulator-py src/simulator/simulation.py
//   transmissibilities :52-74, pressure step :867-904, matrix :1546-1580,
//   right-hand side :1582-1620, well terms :1622-1660, saturation :968-1544;
//   src/simulator/fluid.py relperm :224-248/:377-435, densities :129-158/:330-375,
//   total compressibility :190-222, capillary pressure :273-296; pvt.py :48-64.
//
// This translation unit is compiled with -fmad=false: every expression keeps the
// reference's operation order and rounding (no fused multiply-add), so the
// assembled system matches the reference's float64 evaluation to the last bit
// wherever the reference's arithmetic is elementwise.
//
// The assembly (K1) and the fluxes (K4a) run in two kernels each: the first
// evaluates every cell's phase properties once (a few hundred FP64 instructions),
// the second reads a cell's and its six neighbours' through L1 and L2.
#include "model.cuh"
#include <algorithm>
#include <math.h>
#include <mutex>

namespace impes {

namespace {

constexpr int kPvtCols = 9;  // P, Bo, Bw, Bg, mu_o, mu_w, mu_g, Rs, Rv
enum { C_P = 0, C_BO = 1, C_BW = 2, C_BG = 3, C_MUO = 4, C_MUW = 5, C_MUG = 6, C_RS = 7, C_RV = 8 };

// torch's scalar-exponent pow special cases (x*x, x*x*x, 1/sqrt, 1/x, 1/(x*x)).
__device__ __forceinline__ double tpow(double x, double e) {
  if (e == 0.0) return 1.0;
  if (e == 1.0) return x;
  if (e == 2.0) return x * x;
  if (e == 3.0) return x * x * x;
  if (e == -0.5) return 1.0 / sqrt(x);
  if (e == -1.0) return 1.0 / x;
  if (e == -2.0) return 1.0 / (x * x);
  if (x == 1.0) return 1.0;            // the end points of a saturation range, as pow gives them
  if (x == 0.0 && e > 0.0) return 0.0;
  return pow(x, e);
}
// torch.clamp semantics (NaN passes through; lo > hi yields hi).
__device__ __forceinline__ double tclamp(double x, double lo, double hi) {
  double y = (x < lo) ? lo : x;
  return (y > hi) ? hi : y;
}
__device__ __forceinline__ double tclamp_min(double x, double lo) { return (x < lo) ? lo : x; }
__device__ __forceinline__ double tclamp_max(double x, double hi) { return (x > hi) ? hi : x; }
// torch.maximum: NaN-propagating.
__device__ __forceinline__ double tmaximum(double a, double b) {
  if (isnan(a) || isnan(b)) return __longlong_as_double(0x7ff8000000000000LL);
  return a > b ? a : b;
}

// PVT table staged in shared memory: columns [9][rows] and slopes [8][rows-1].
struct PvtSmem {
  int rows;
  const double* col;    // 9 * rows
  const double* slope;  // 8 * (rows - 1)
};

// The table as the kernels stage it: columns [9][rows], then slopes [8][rows - 1]
// of the columns after the pressure.
__global__ void k_pvt_table(int rows, const double* __restrict__ g, double* __restrict__ tab) {
  for (int t = threadIdx.x; t < rows * kPvtCols; t += blockDim.x) tab[(t % kPvtCols) * rows + t / kPvtCols] = g[t];
  for (int t = threadIdx.x; t < (kPvtCols - 1) * (rows - 1); t += blockDim.x) {
    const int c = 1 + t / (rows - 1), r = t % (rows - 1);
    tab[kPvtCols * rows + t] = (g[(r + 1) * kPvtCols + c] - g[r * kPvtCols + c]) /
                               (g[(r + 1) * kPvtCols] - g[r * kPvtCols]);
  }
}
__device__ void pvt_stage(const double* __restrict__ tab, int rows, double* s_col, double* s_slope) {
  for (int t = threadIdx.x; t < kPvtCols * rows; t += blockDim.x) s_col[t] = tab[t];
  for (int t = threadIdx.x; t < (kPvtCols - 1) * (rows - 1); t += blockDim.x) s_slope[t] = tab[kPvtCols * rows + t];
  __syncthreads();
}

// numpy.interp(x, xp, fp) with flat extrapolation (pvt.py:48-50), in two parts:
// where x lies in the table (searched once for all columns read there) and the
// value of a column.
struct PvtAt {
  double x;
  int lo;       // interval, or the row whose value is taken
  int kind;     // 0: interpolate, 1: row lo, 2: x is NaN
};
__device__ PvtAt pvt_find(const PvtSmem& t, double x) {
  const int n = t.rows;
  const double* xp = t.col;
  if (isnan(x)) return {x, 0, 2};
  if (x < xp[0]) return {x, 0, 1};
  if (x >= xp[n - 1]) return {x, n - 1, 1};
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (xp[mid] <= x) lo = mid; else hi = mid;
  }
  return {x, lo, xp[lo] == x ? 1 : 0};
}
// pvt_find for an x near one found before: its interval is tried first
__device__ PvtAt pvt_find_near(const PvtSmem& t, double x, const PvtAt& near) {
  const int lo = near.lo;
  if (near.kind != 2 && lo < t.rows - 1 && t.col[lo] < x && x < t.col[lo + 1]) return {x, lo, 0};
  return pvt_find(t, x);
}
__device__ __forceinline__ double pvt_val(const PvtSmem& t, int c, const PvtAt& a) {
  const int n = t.rows, lo = a.lo;
  const double* xp = t.col;
  const double* fp = t.col + c * n;
  if (a.kind == 2) return a.x;
  if (a.kind == 1) return fp[lo];
  const double sl = t.slope[(c - 1) * (n - 1) + lo];
  double r = sl * (a.x - xp[lo]) + fp[lo];
  if (isnan(r)) {
    r = sl * (a.x - xp[lo + 1]) + fp[lo + 1];
    if (isnan(r) && fp[lo] == fp[lo + 1]) r = fp[lo];
  }
  return r;
}
// Fluid._eval_pvt(p, key): interpolation at p / 1e6 MPa (fluid.py:186-187).
__device__ __forceinline__ PvtAt pvt_at(const ModelParams& P, const PvtSmem& t, double p_pa) {
  if (P.pvt_rows == 0) return {0.0, 0, 1};
  return pvt_find(t, p_pa / 1e6);
}

struct KR { double kro, krw, krg; };

// Fluid.get_rel_perms(sw, sg) (fluid.py:231-248, 377-435).
__device__ KR relperms(const ModelParams& P, double sw, double sg) {
  KR r;
  const double den = (1 - P.sw_cr) - P.so_r;
  double s_norm = tclamp((sw - P.sw_cr) / den, 0.0, 1.0);
  r.krw = tpow(s_norm, P.nw);
  if (P.relperm_model == 1) {
    const double dw = (1.0 - P.sw_cr) - P.so_r;
    double swn = tclamp((sw - P.sw_cr) / (dw + 1e-12), 0.0, 1.0);
    const double dg = (1.0 - P.sg_cr) - P.so_r;
    double sgn = tclamp((sg - P.sg_cr) / (dg + 1e-12), 0.0, 1.0);
    double krow = P.ko_end_w * tpow(1.0 - swn, P.now);
    double krog = P.ko_end_g * tpow(1.0 - sgn, P.nog);
    double kmin = P.ko_end_w < P.ko_end_g ? P.ko_end_w : P.ko_end_g;
    r.kro = tclamp_min(krow + krog - kmin, 0.0);
  } else {
    r.kro = tpow(1 - s_norm, P.no);
  }
  double sgn2 = tclamp(sg / ((1.0 - P.sw_cr) - P.so_r + 1e-10), 0.0, 1.0);
  r.krg = tpow(sgn2, P.ng);
  return r;
}

struct Visc { double o, w, g; };
__device__ __forceinline__ Visc viscosities(const ModelParams& P, const PvtSmem& t, const PvtAt& at) {
  Visc v;
  if (P.pvt_rows > 0) {
    v.o = pvt_val(t, C_MUO, at) * 1e-3;
    v.w = pvt_val(t, C_MUW, at) * 1e-3;
    v.g = pvt_val(t, C_MUG, at) * 1e-3;
  } else {
    v.o = P.mu_o; v.w = P.mu_w; v.g = P.mu_g;
  }
  return v;
}

struct Rho { double w, o, g; };
// Fluid.rho_w / rho_o / rho_g at pressure p (fluid.py:129-158, 330-375).
__device__ __forceinline__ Rho densities(const ModelParams& P, const PvtSmem& t, double p, const PvtAt& at) {
  Rho r;
  if (P.pvt_rows > 0) {
    double bw = pvt_val(t, C_BW, at), bo = pvt_val(t, C_BO, at), rs = pvt_val(t, C_RS, at);
    double bg = pvt_val(t, C_BG, at), rv = pvt_val(t, C_RV, at);
    r.w = P.rho_w_ref / (bw + 1e-12);
    r.o = (P.rho_o_ref + rs * P.rho_g_ref) / (bo + 1e-12);
    r.g = (P.rho_g_ref + rv * P.rho_o_ref) / (bg + 1e-12);
  } else {
    r.w = P.rho_w_ref * (1.0 + P.c_w * (p - 1e5));
    r.o = P.rho_o_ref * (1.0 + P.c_o * (p - 1e5));
    r.g = P.rho_g_ref * (1.0 + P.c_g * (p - 1e5));
  }
  return r;
}

// calc_total_compressibility (fluid.py:190-222).
__device__ __forceinline__ double total_compressibility(const ModelParams& P, const PvtSmem& t, double sw, double sg,
                                                        const PvtAt& at) {
  if (P.pvt_rows == 0) return P.cf;
  const double P_mpa = at.x;            // p / 1e6
  const double Pp = P_mpa + 0.1, Pm = P_mpa - 0.1;
  const PvtAt a0 = pvt_find_near(t, P_mpa * 1e6 / 1e6, at);
  const PvtAt ap = pvt_find_near(t, Pp * 1e6 / 1e6, a0), am = pvt_find_near(t, Pm * 1e6 / 1e6, a0);
  double c[3];
  const int cols[3] = {C_BW, C_BO, C_BG};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double B = pvt_val(t, cols[q], a0), Bp = pvt_val(t, cols[q], ap), Bm = pvt_val(t, cols[q], am);
    double dB = (Bp - Bm) / (2 * 0.1);
    c[q] = -(dB / (B + 1e-12)) / 1e6;
  }
  const double so = 1.0 - sw - sg;
  return P.c_r + sw * c[0] + so * c[1] + sg * c[2];
}

__device__ __forceinline__ double capillary(const ModelParams& P, double sw) {
  if (P.pc_scale == 0.0) return 0.0;
  double s_norm = tclamp((sw - P.sw_cr) / ((1 - P.sw_cr) - P.so_r), 0.0, 1.0);
  return P.pc_scale * tpow(1.0 - s_norm + 1e-6, -P.pc_exponent);
}
__device__ __forceinline__ double capillary_og(const ModelParams& P, double sg) {
  if (P.pc_og_scale == 0.0) return 0.0;
  const double denom = (1 - P.sw_cr) - P.so_r;
  double sgn = tclamp(sg / (denom + 1e-12), 0.0, 1.0);
  return P.pc_og_scale * tpow(1.0 - sgn + 1e-6, -P.pc_og_exponent);
}

// Binary search of `cell` in the sorted distinct well-cell list.
__device__ __forceinline__ int well_slot(const int* wc, int nwc, int cell) {
  int lo = 0, hi = nwc - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    int v = wc[mid];
    if (v == cell) return mid;
    if (v < cell) lo = mid + 1; else hi = mid - 1;
  }
  return -1;
}

// ------------------------------------------------------------ static data
__global__ void k_transmissibility(ModelParams P, const double* __restrict__ kx,
                                   const double* __restrict__ ky, const double* __restrict__ kz,
                                   const double* __restrict__ poro, double* tx, double* ty,
                                   double* tz, double* pv) {
  const long long N = P.N;
  const double cell_volume = (P.dx * P.dy) * P.dz;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N;
       c += (long long)gridDim.x * blockDim.x) {
    int k = c % P.nz;
    long long r = c / P.nz;
    int j = r % P.ny;
    int i = r / P.ny;
    pv[c] = cell_volume * poro[c];
    if (i < P.nx - 1) {
      double a = kx[c], b = kx[c + (long long)P.ny * P.nz];
      tx[c] = 2 * a * b / (a + b + 1e-15) * P.dy * P.dz / P.dx;          // simulation.py:66-67
    }
    if (j < P.ny - 1) {
      double a = ky[c], b = ky[c + P.nz];
      ty[((long long)i * (P.ny - 1) + j) * P.nz + k] = 2 * a * b / (a + b + 1e-15) * P.dx * P.dz / P.dy;
    }
    if (k < P.nz - 1) {
      double a = kz[c], b = kz[c + 1];
      tz[((long long)i * P.ny + j) * (P.nz - 1) + k] = 2 * a * b / (a + b + 1e-15) * P.dx * P.dy / P.dz;
    }
  }
}

__global__ void k_pattern(ModelParams P, int nnz, int* rowptr, int* col) {
  const int plane = P.ny * P.nz;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c <= P.N;
       c += (long long)gridDim.x * blockDim.x) {
    if (c == P.N) { rowptr[c] = nnz; continue; }
    const int i = (int)c / plane, r = (int)c - i * plane, j = r / P.nz, k = r - j * P.nz;
    int e = pattern_row((int)c, i, j, k, P.nx, P.ny, P.nz);
    rowptr[c] = e;
    if (i > 0) col[e++] = (int)(c - plane);
    if (j > 0) col[e++] = (int)(c - P.nz);
    if (k > 0) col[e++] = (int)(c - 1);
    col[e++] = (int)c;
    if (k < P.nz - 1) col[e++] = (int)(c + 1);
    if (j < P.ny - 1) col[e++] = (int)(c + P.nz);
    if (i < P.nx - 1) col[e++] = (int)(c + plane);
  }
}

// Items that wells bring along are dealt over the blocks, then over a block's warps,
// then over their lanes: items block, block + grid, .. of thread 0, of thread 32, ..
// and so on, in steps of the launch.  On a large grid a warp has one at most (all of
// them in one block were its critical path); a grid of one block has its 256 threads
// work on them (one thread a block took 2.3 ms for 120 wells of a 16 x 16 model).
__device__ __forceinline__ int dealt_first() {
  return ((threadIdx.x & 31) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * gridDim.x + blockIdx.x;
}

// The kernels over cells take them in runs of kCells consecutive ones, a thread
// each; wells are looked up only in a run that holds a well's cell.
constexpr int kCells = 256;
__device__ __forceinline__ bool run_has_well(const int* wc, int nwc, int c0) {
  int lo = 0, hi = nwc;                 // first well cell at or after c0
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (wc[mid] < c0) lo = mid + 1; else hi = mid;
  }
  return lo < nwc && wc[lo] < c0 + kCells;
}

// ------------------------------------------------------------ K1 assembly
// K1a: per cell (simulation.py:870-882) the total mobility mt, the gravity sum
// gs = sum of mobility x density, the oil mobility mo, the capillary pressure pc
// (the last three where the right-hand side reads them) and the accumulation
// coefficient acc = PV ct / dt (simulation.py:1569-1576).
// Bound by FP64 and integer instructions, about 900 a cell: 85 us at 1e6 cells.  Evaluated in bricks
// with a one-cell halo in shared memory, every cell's properties were computed
// 2.0 times and indexed with runtime divisions: 5,800 instructions a cell,
// 268 us at 1e6 cells for the whole assembly.
__global__ void __launch_bounds__(kCells) k_cell_props(
    ModelParams P, const double* __restrict__ pvt_g, const double* __restrict__ p, const double* __restrict__ sw,
    const double* __restrict__ sg, const double* __restrict__ pv, double dt, double* __restrict__ mt,
    double* __restrict__ gs, double* __restrict__ mo, double* __restrict__ pc, double* __restrict__ acc) {
  __shared__ double s_col[kPvtCols * kMaxPvtRows];
  __shared__ double s_slope[(kPvtCols - 1) * kMaxPvtRows];
  PvtSmem T{P.pvt_rows, s_col, s_slope};
  if (P.pvt_rows > 0) pvt_stage(pvt_g, P.pvt_rows, s_col, s_slope);
  const bool grav = (P.dz > 0) && (P.nz > 1);
  for (int c = blockIdx.x * kCells + threadIdx.x; c < P.N; c += gridDim.x * kCells) {
    const double p_ = p[c], swc = sw[c], sgc = sg[c];
    const KR kr = relperms(P, swc, sgc);
    const PvtAt at = pvt_at(P, T, p_);
    const Visc mu = viscosities(P, T, at);
    const double w = kr.krw / mu.w, o = kr.kro / mu.o, g = kr.krg / mu.g;
    mt[c] = w + o + g;
    if (grav) {
      const Rho r = densities(P, T, p_, at);
      gs[c] = w * r.w + o * r.o + g * r.g;
    }
    if (P.pc_scale > 0) {
      mo[c] = o;
      pc[c] = capillary(P, swc);
    }
    const double ct = total_compressibility(P, T, swc, sgc, at);
    acc[c] = pv[c] * ct / dt;
  }
}

// K1b: one matrix row and right-hand side entry per cell, from its and its
// neighbours' properties.  A run's matrix values are one contiguous piece of the
// CSR array: rows are put together in shared memory and stored from there.
// Bound by the loads' latency and the 10 doubles a row writes and reads: 54 us at 1e6
// cells.
__global__ void __launch_bounds__(kCells, 3) k_assemble(
    ModelParams P, const double* __restrict__ p, const double* __restrict__ mt, const double* __restrict__ gs,
    const double* __restrict__ mo, const double* __restrict__ pc, const double* __restrict__ acc,
    const double* __restrict__ tx, const double* __restrict__ ty, const double* __restrict__ tz,
    const WellDev* __restrict__ wells, const int* __restrict__ wc_cells,
    const int* __restrict__ wc_ptr, const int* __restrict__ wc_wells, int* __restrict__ well_mode,
    double* __restrict__ val, double* __restrict__ rhs) {
  __shared__ double s_val[7 * kCells];
  __shared__ int s_e0, s_e1;
  const bool grav = (P.dz > 0) && (P.nz > 1);
  const int plane = P.ny * P.nz;
  for (int c0 = blockIdx.x * kCells; c0 < P.N; c0 += gridDim.x * kCells) {
    const int c = c0 + threadIdx.x;
    const bool has_well = P.nwc > 0 && run_has_well(wc_cells, P.nwc, c0);
    const int last = min(c0 + kCells, P.N) - 1;
    int e = 0, entries = 0;
    double row[7];
    if (c <= last) {
      const int i = c / plane, r = c - i * plane, j = r / P.nz, k = r - j * P.nz;
      const bool hxm = i > 0, hxp = i < P.nx - 1, hym = j > 0, hyp = j < P.ny - 1;
      const bool hzm = k > 0, hzp = k < P.nz - 1;
      // the face arrays (one cell less along their own direction)
      const int iy = c - i * P.nz, iz = c - (i * P.ny + j);
      const bool have[6] = {hxp, hxm, hyp, hym, hzp, hzm};
      const int nb[6] = {c + plane, c - plane, c + P.nz, c - P.nz, c + 1, c - 1};
      const double t_[6] = {hxp ? tx[c] : 0.0, hxm ? tx[c - plane] : 0.0, hyp ? ty[iy] : 0.0,
                            hym ? ty[iy - P.nz] : 0.0, hzp ? tz[iz] : 0.0, hzm ? tz[iz - 1] : 0.0};
      const double p0 = p[c], mt0 = mt[c];
      double pn[6], mn[6];
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        pn[d] = have[d] ? p[nb[d]] : 0.0;
        mn[d] = have[d] ? mt[nb[d]] : 0.0;
      }
      // total-mobility transmissibility of a face, upwind by the pressure of its
      // lower cell against its upper one (simulation.py:885-895); up[d]: the
      // upwind side is this cell
      bool up[6];
      double tf[6];
#pragma unroll
      for (int d = 0; d < 6; ++d) {
        const bool plus = d % 2 == 0;            // this cell is the lower one
        const double dp = plus ? p0 - pn[d] : pn[d] - p0;
        up[d] = plus ? dp > 0 : !(dp > 0);
        tf[d] = have[d] ? t_[d] * (up[d] ? mt0 : mn[d]) : 0.0;
      }

      // wells at this cell (simulation.py:1622-1660), in configuration order
      double well_diag = 0.0, q_well = 0.0;
      if (has_well) {
        const int slot = well_slot(wc_cells, P.nwc, c);
        if (slot >= 0) {
          for (int q = wc_ptr[slot]; q < wc_ptr[slot + 1]; ++q) {
            int w = wc_wells[q];
            const WellDev W = wells[w];
            if (W.control_bhp == 0) {
              double rate_si = (W.value * P.rate_scale) / 86400.0 * (W.is_injector ? 1 : -1);
              if (!W.is_injector && W.has_bhp_min) {
                double denom = W.well_index * mt0 + 1e-12;
                double p_req = p0 - rate_si / denom;
                double p_min = W.bhp_min * 1e6;
                if (p_req < p_min) {
                  well_mode[w] = 1;
                  well_diag += W.well_index * mt0;
                  q_well += W.well_index * mt0 * p_min;
                  continue;
                }
              }
              well_mode[w] = 0;
              q_well += rate_si;
            } else {
              well_diag += W.well_index * mt0;
              q_well += W.well_index * mt0 * (W.value * 1e6);
            }
          }
        }
      }

      // diagonal in the reference's scatter_add order: x+, x-, y+, y-, z+, z-
      const double acc0 = acc[c];
      double diag = 0.0;
#pragma unroll
      for (int d = 0; d < 6; ++d)
        if (have[d]) diag += tf[d];
      diag += acc0;
      diag += well_diag;

      // row in CSR order: x-, y-, z-, diag, z+, y+, x+
      e = pattern_row(c, i, j, k, P.nx, P.ny, P.nz);
      row[0] = -tf[1]; row[1] = -tf[3]; row[2] = -tf[5]; row[3] = diag;
      row[4] = -tf[4]; row[5] = -tf[2]; row[6] = -tf[0];
      entries = (hxm ? 1 : 0) | (hym ? 2 : 0) | (hzm ? 4 : 0) | 8 | (hzp ? 16 : 0) | (hyp ? 32 : 0) | (hxp ? 64 : 0);

      // right-hand side (simulation.py:1582-1620)
      const double comp = acc0 * p0;
      double qg = 0.0;
      if (grav) {
        const double gs0 = gs[c];
        if (hzp) qg -= t_[4] * P.gravity * P.dz * (up[4] ? gs0 : gs[c + 1]);
        if (hzm) qg += t_[5] * P.gravity * P.dz * (up[5] ? gs0 : gs[c - 1]);
      }
      double qpc = 0.0;
      if (P.pc_scale > 0) {
        const double mo0 = mo[c], pc0 = pc[c];
        // the reference's order: x-, x+, y-, y+, z-, z+
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const int d = q ^ 1;
          if (!have[d]) continue;
          const double m = up[d] ? mo0 : mo[nb[d]];
          if (d % 2) qpc += t_[d] * m * (pc0 - pc[nb[d]]);
          else qpc -= t_[d] * m * (pc[nb[d]] - pc0);
        }
      }
      rhs[c] = comp + q_well + qg + qpc;
      if (c == c0) s_e0 = e;
      if (c == last) s_e1 = e + __popc(entries);
    }
    __syncthreads();
    if (entries) {
      int at = e - s_e0;
#pragma unroll
      for (int d = 0; d < 7; ++d)
        if (entries >> d & 1) s_val[at++] = row[d];
    }
    __syncthreads();
    for (int x = threadIdx.x; x < s_e1 - s_e0; x += kCells) val[s_e0 + x] = s_val[x];
    __syncthreads();
  }
}

// ------------------------------------------------ K4: saturation update
// Well sources of the saturation step (simulation.py:1044-1347), one thread,
// wells in configuration order; component balance of the step (non-substep part).
__device__ void well_cell_phase(const ModelParams& P, const PvtSmem& T, double p, double sw,
                                double sg, double& mt, double& fw, double& fg, double& fo) {
  KR kr = relperms(P, sw, sg);
  Visc mu = viscosities(P, T, pvt_at(P, T, p));
  double mw = kr.krw / mu.w, mo = kr.kro / mu.o, mg = kr.krg / mu.g;
  mt = mw + mo + mg;
  fw = mw / (mt + 1e-10);
  fg = mg / (mt + 1e-10);
  fo = mo / (mt + 1e-10);
}

// What a well adds: to the (water, gas, oil) sources of its cell and to the
// component balance (oil in, oil out, gas in, gas out); bit k of mask marks
// addition k as made.
struct WellTerms {
  double q[3], b[4];
  int mask, pad;
};
struct WellArgs {
  const WellDev* wells;
  const int *wc_cells, *wc_ptr, *wc_wells;
  WellTerms* terms;    // per well
  double* state;       // per well cell: Sw, Sg and their increments before the substeps
  double* bal;         // 12 balances
  double* well_q;
  double* well_rates;
};
// A well's terms, by one thread (they depend only on its cell's state).
__device__ __noinline__ void well_source(const ModelParams& P, const PvtSmem& T, const WellArgs& A, int w,
                                         const double* __restrict__ p_new, const double* __restrict__ sw,
                                         const double* __restrict__ sg, const double* __restrict__ pv, double dt) {
  double *well_q = A.well_q, *well_rates = A.well_rates;
  const bool pvt = P.pvt_rows > 0;
  const double so_r = P.so_r, sw_min = P.sw_cr, sg_min = P.sg_cr;
  {
    const WellDev W = A.wells[w];
    const int c = W.cell;
    int mask = 0;
    double dq[3] = {0.0, 0.0, 0.0}, db[4] = {0.0, 0.0, 0.0, 0.0};
    if (c >= 0) {  // a well outside the grid contributes nothing (simulation.py:1053-1054)
      const double p = p_new[c], sw_c = sw[c], sg_c = sg[c], pv_c = pv[c];
      double mt, fw_, fg_, fo_;
      well_cell_phase(P, T, p, sw_c, sg_c, mt, fw_, fg_, fo_);
      double Bo = 0, Bw = 0, Bg = 0, Rs = 0, Rv = 0;
      if (pvt) {
        const PvtAt at = pvt_at(P, T, p);
        Bo = pvt_val(T, C_BO, at); Bw = pvt_val(T, C_BW, at); Bg = pvt_val(T, C_BG, at);
        Rs = pvt_val(T, C_RS, at); Rv = pvt_val(T, C_RV, at);
      }
      if (W.control_bhp == 0) {
        const double q_base = (W.value * P.rate_scale) / 86400.0;
        double q_total;
        if (W.is_injector && W.surface_rate && pvt)
          q_total = q_base * (W.injected_phase == 1 ? Bg : Bw);
        else
          q_total = q_base;
        q_total *= (W.is_injector ? 1 : -1);
        if (W.is_injector) {
          if (W.injected_phase == 1) {
            double sg_up = fmax(0.0, (1.0 - so_r - sw_c) - sg_c);
            double dS = (dt / fmax(pv_c, 1e-12)) * q_total;
            double alpha = 1.0;
            if (dS > 0.0) alpha = fmin(alpha, sg_up / fmax(dS, 1e-12));
            else alpha = fmin(alpha, (sg_c - sg_min) / fmax(fabs(dS), 1e-12));
            q_total *= fmax(0.0, fmin(1.0, alpha));
            dq[1] = q_total; mask |= 2;
            if (pvt) {
              double qg_surf = fmax(q_total, 0.0) / fmax(Bg, 1e-12) * 86400.0;
              double scale = dt / 86400.0;
              db[2] = qg_surf * scale;        // gas in
              db[0] = Rv * qg_surf * scale;   // oil in
              mask |= 8 | 32;
            }
          } else {
            double sw_up = fmax(0.0, (1.0 - so_r - sg_c) - sw_c);
            double dS = (dt / fmax(pv_c, 1e-12)) * q_total;
            double alpha = 1.0;
            if (dS > 0.0) alpha = fmin(alpha, sw_up / fmax(dS, 1e-12));
            else alpha = fmin(alpha, (sw_c - sw_min) / fmax(fabs(dS), 1e-12));
            q_total *= fmax(0.0, fmin(1.0, alpha));
            dq[0] = q_total; mask |= 1;
          }
        } else {
          // producer at rate
          if (pvt) {
            if (W.surface_rate) {
              switch (W.surface_phase) {
                case 0: q_total = -(q_base / fmax(fo_ / fmax(Bo, 1e-12) + fg_ * Rv / fmax(Bg, 1e-12), 1e-12)); break;
                case 1: q_total = -(q_base * Bw) / fmax(fw_, 1e-8); break;
                case 2: q_total = -(q_base / fmax(fg_ / fmax(Bg, 1e-12) + fo_ * Rs / fmax(Bo, 1e-12), 1e-12)); break;
                default:
                  q_total = -(q_base / fmax(fo_ / fmax(Bo, 1e-12) + fg_ * Rv / fmax(Bg, 1e-12) +
                                                fw_ / fmax(Bw, 1e-12), 1e-12));
              }
            }
            double sw_up = fmax(0.0, (1.0 - so_r - sg_c) - sw_c);
            double sw_dn = fmax(0.0, sw_c - sw_min);
            double sg_up = fmax(0.0, (1.0 - so_r - sw_c) - sg_c);
            double sg_dn = fmax(0.0, sg_c - sg_min);
            double dSw = (dt / fmax(pv_c, 1e-12)) * (q_total * fw_);
            double dSg = (dt / fmax(pv_c, 1e-12)) * (q_total * fg_);
            double alpha = 1.0;
            alpha = dSw > 0.0 ? fmin(alpha, sw_up / fmax(dSw, 1e-12)) : fmin(alpha, sw_dn / fmax(fabs(dSw), 1e-12));
            alpha = dSg > 0.0 ? fmin(alpha, sg_up / fmax(dSg, 1e-12)) : fmin(alpha, sg_dn / fmax(fabs(dSg), 1e-12));
            alpha = fmax(0.0, fmin(1.0, alpha));
            q_total *= alpha;
            if (W.limit_mask) {
              double d_o = fo_ / fmax(Bo, 1e-12) + fg_ * Rv / fmax(Bg, 1e-12);
              double d_w = fw_ / fmax(Bw, 1e-12);
              double d_g = fg_ / fmax(Bg, 1e-12) + fo_ * Rs / fmax(Bo, 1e-12);
              double d_l = d_o + d_w;
              double mx = INFINITY;
              bool any = false;
              if ((W.limit_mask & 1) && d_o > 0) { mx = fmin(mx, (W.limits[0] / 86400.0) / d_o); any = true; }
              if ((W.limit_mask & 2) && d_w > 0) { mx = fmin(mx, (W.limits[1] / 86400.0) / d_w); any = true; }
              if ((W.limit_mask & 4) && d_g > 0) { mx = fmin(mx, (W.limits[2] / 86400.0) / d_g); any = true; }
              if ((W.limit_mask & 8) && d_l > 0) { mx = fmin(mx, (W.limits[3] / 86400.0) / d_l); any = true; }
              if (any && fabs(q_total) > mx) q_total = -mx;
            }
            double aq = fabs(q_total);
            double oil_s = aq * (fo_ / fmax(Bo, 1e-12) + fg_ * Rv / fmax(Bg, 1e-12)) * 86400.0;
            double wat_s = aq * (fw_ / fmax(Bw, 1e-12)) * 86400.0;
            double gas_s = aq * (fg_ / fmax(Bg, 1e-12) + fo_ * Rs / fmax(Bo, 1e-12)) * 86400.0;
            well_rates[4 * w + 0] = oil_s;
            well_rates[4 * w + 1] = wat_s;
            well_rates[4 * w + 2] = gas_s;
            well_rates[4 * w + 3] = oil_s + wat_s;
            well_q[w] = q_total;
            double qo_res = -q_total * fo_, qg_res = -q_total * fg_;
            db[1] = dt * (fmax(qo_res, 0.0) / fmax(Bo, 1e-12) + Rv * fmax(qg_res, 0.0) / fmax(Bg, 1e-12));
            db[3] = dt * (fmax(qg_res, 0.0) / fmax(Bg, 1e-12) + Rs * fmax(qo_res, 0.0) / fmax(Bo, 1e-12));
            mask |= 16 | 64;
          }
          dq[0] = q_total * fw_;
          dq[1] = q_total * fg_;
          dq[2] = q_total * fo_;
          mask |= 1 | 2 | 4;
        }
      } else {
        const double p_bhp = W.value * 1e6;
        const double q_total = W.well_index * mt * (p - p_bhp);
        if (W.is_injector) {
          if (W.injected_phase == 1) {
            dq[1] = -q_total; mask |= 2;
            if (pvt) {
              double qg_surf = fmax(-q_total, 0.0) / fmax(Bg, 1e-12) * 86400.0;
              double scale = dt / 86400.0;
              db[2] = qg_surf * scale;
              db[0] = Rv * qg_surf * scale;
              mask |= 8 | 32;
            }
          } else {
            dq[0] = -q_total; mask |= 1;
          }
        } else {
          dq[0] = (-q_total) * fw_;
          dq[1] = (-q_total) * fg_;
          dq[2] = (-q_total) * fo_;
          mask |= 1 | 2 | 4;
          if (pvt) {
            double qabs = fabs(q_total);
            double qo_res = qabs * fo_, qg_res = qabs * fg_;
            db[1] = dt * (qo_res / fmax(Bo, 1e-12) + Rv * qg_res / fmax(Bg, 1e-12));
            db[3] = dt * (qg_res / fmax(Bg, 1e-12) + Rs * qo_res / fmax(Bo, 1e-12));
            mask |= 16 | 64;
          }
        }
      }
    }
    WellTerms& t = A.terms[w];
    t.mask = mask;
    for (int k = 0; k < 3; ++k) t.q[k] = dq[k];
    for (int k = 0; k < 4; ++k) t.b[k] = db[k];
  }
}

// K4a: fluxes, divergence, dS and the substep ratio (simulation.py:968-1042, 1351-1379).
// K4a': water and gas mobilities and densities and the oil-gas capillary pressure
// of every cell, at the new pressure; and the wells' terms.
__global__ void __launch_bounds__(kCells, 4) k_flux_props(
    ModelParams P, const double* __restrict__ pvt_g, const double* __restrict__ p, const double* __restrict__ sw,
    const double* __restrict__ sg, const double* __restrict__ pv, double dt, double* __restrict__ mw,
    double* __restrict__ mg, double* __restrict__ rw, double* __restrict__ rg, double* __restrict__ pcg, WellArgs A,
    const int* pred) {
  if (pred && *pred == 0) return;
  __shared__ double s_col[kPvtCols * kMaxPvtRows];
  __shared__ double s_slope[(kPvtCols - 1) * kMaxPvtRows];
  PvtSmem T{P.pvt_rows, s_col, s_slope};
  if (P.pvt_rows > 0) pvt_stage(pvt_g, P.pvt_rows, s_col, s_slope);
  for (int w = dealt_first(); w < P.nwells; w += blockDim.x * gridDim.x)
    well_source(P, T, A, w, p, sw, sg, pv, dt);
  const bool grav = (P.dz > 0) && (P.nz > 1);
  for (int c = blockIdx.x * kCells + threadIdx.x; c < P.N; c += gridDim.x * kCells) {
    const double p_ = p[c], swc = sw[c], sgc = sg[c];
    const KR kr = relperms(P, swc, sgc);
    const PvtAt at = pvt_at(P, T, p_);
    const Visc mu = viscosities(P, T, at);
    mw[c] = kr.krw / mu.w;
    mg[c] = kr.krg / mu.g;
    if (grav) {
      const Rho r = densities(P, T, p_, at);
      rw[c] = r.w;
      rg[c] = r.g;
    }
    if (P.pc_og_scale > 0) pcg[c] = capillary_og(P, sgc);
  }
}

__global__ void __launch_bounds__(kCells, 3) k_saturation_flux(
    ModelParams P, const double* __restrict__ p, const double* __restrict__ mw, const double* __restrict__ mg,
    const double* __restrict__ rw, const double* __restrict__ rg, const double* __restrict__ pcg,
    const double* __restrict__ sw, const double* __restrict__ sg, const double* __restrict__ tx,
    const double* __restrict__ ty, const double* __restrict__ tz, const double* __restrict__ pv,
    WellArgs A, double dt, double* __restrict__ dsw_out, double* __restrict__ dsg_out,
    double* __restrict__ red, unsigned* __restrict__ counter, int* __restrict__ nsub_out, const int* pred) {
  if (pred && *pred == 0) return;
  __shared__ double s_red[3 * 8];
  __shared__ bool s_last;
  const bool grav = (P.dz > 0) && (P.nz > 1);
  const bool pcog = P.pc_og_scale > 0;
  const int plane = P.ny * P.nz;
  double rmax = 0.0, rnan = 0.0, rinf = 0.0;
  for (int c0 = blockIdx.x * kCells; c0 < P.N; c0 += gridDim.x * kCells) {
    const bool has_well = P.nwc > 0 && run_has_well(A.wc_cells, P.nwc, c0);
    const int c = c0 + threadIdx.x;
    if (c >= P.N) continue;
    const int i = c / plane, r = c - i * plane, j = r / P.nz, k = r - j * P.nz;
    const int iy = c - i * P.nz, iz = c - (i * P.ny + j);
    // the reference's order of a cell's faces: x+, x-, y+, y-, z+, z-
    const bool have[6] = {i < P.nx - 1, i > 0, j < P.ny - 1, j > 0, k < P.nz - 1, k > 0};
    const int nb[6] = {c + plane, c - plane, c + P.nz, c - P.nz, c + 1, c - 1};
    const double t_[6] = {have[0] ? tx[c] : 0.0, have[1] ? tx[c - plane] : 0.0, have[2] ? ty[iy] : 0.0,
                          have[3] ? ty[iy - P.nz] : 0.0, have[4] ? tz[iz] : 0.0, have[5] ? tz[iz - 1] : 0.0};
    const double p0 = p[c], mw0 = mw[c], mg0 = mg[c];
    double pn[6], wn[6], gn[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      pn[d] = have[d] ? p[nb[d]] : 0.0;
      wn[d] = have[d] ? mw[nb[d]] : 0.0;
      gn[d] = have[d] ? mg[nb[d]] : 0.0;
    }
    const double rw0 = grav ? rw[c] : 0.0, rg0 = grav ? rg[c] : 0.0, pcg0 = pcog ? pcg[c] : 0.0;
    double dw = 0.0, dg = 0.0;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      if (!have[d]) continue;
      const bool plus = d % 2 == 0;              // this cell is the face's lower one
      const double dp = plus ? p0 - pn[d] : pn[d] - p0;
      const bool up = plus ? dp > 0 : !(dp > 0); // the upwind side is this cell
      const double m_w = up ? mw0 : wn[d], m_g = up ? mg0 : gn[d];
      double pw = dp, pg = dp;
      if (d >= 4 && grav) {
        const double rwn = rw[nb[d]], rgn = rg[nb[d]];
        const double rwa = 0.5 * (plus ? rw0 + rwn : rwn + rw0);
        const double rga = 0.5 * (plus ? rg0 + rgn : rgn + rg0);
        pw = dp + P.gravity * rwa * P.dz;
        pg = dp + P.gravity * rga * P.dz;
      }
      const double fw = t_[d] * m_w * pw;
      double fg;
      if (pcog) {
        const double pcn = pcg[nb[d]];
        fg = t_[d] * m_g * (pg - (plus ? pcn - pcg0 : pcg0 - pcn));
      } else {
        fg = t_[d] * m_g * pg;
      }
      if (plus) { dw += fw; dg += fg; }
      else { dw -= fw; dg -= fg; }
    }
    double qwc = 0.0, qgc = 0.0;
    int slot = -1;
    if (has_well) {
      slot = well_slot(A.wc_cells, P.nwc, c);
      if (slot >= 0)                   // the cell's wells in configuration order
        for (int q = A.wc_ptr[slot]; q < A.wc_ptr[slot + 1]; ++q) {
          const WellTerms& t = A.terms[A.wc_wells[q]];
          if (t.mask & 1) qwc += t.q[0];
          if (t.mask & 2) qgc += t.q[1];
        }
    }
    const double f = dt / pv[c];
    const double dSw = f * (qwc - dw);
    const double dSg = f * (qgc - dg);
    dsw_out[c] = dSw;
    dsg_out[c] = dSg;
    const double swc = sw[c], sgc = sg[c], eps = 1e-12;
    if (slot >= 0) {
      A.state[4 * slot] = swc;
      A.state[4 * slot + 1] = sgc;
      A.state[4 * slot + 2] = dSw;
      A.state[4 * slot + 3] = dSg;
    }
    const double sw_up = tclamp_min(1.0 - P.so_r - sgc - swc, 0.0);
    const double sw_dn = tclamp_min(swc - P.sw_cr, 0.0);
    const double sg_up = tclamp_min(1.0 - P.so_r - swc - sgc, 0.0);
    const double sg_dn = tclamp_min(sgc - P.sg_cr, 0.0);
    double rw_ = dSw > 0 ? dSw / tclamp_min(sw_up, eps) : (-dSw) / tclamp_min(sw_dn, eps);
    double rg_ = dSg > 0 ? dSg / tclamp_min(sg_up, eps) : (-dSg) / tclamp_min(sg_dn, eps);
    double rl = tmaximum(fabs(dSw) / P.max_dS, fabs(dSg) / P.max_dS);
    double rat = tmaximum(tmaximum(rw_, rg_), rl);
    if (isnan(rat)) rnan = 1.0;
    else if (isinf(rat)) rinf = 1.0;
    else rmax = fmax(rmax, rat);
  }
  // block max -> partials; the last block derives N (simulation.py:1371-1379)
  rmax = warp_max(rmax); rnan = warp_max(rnan); rinf = warp_max(rinf);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { s_red[wid] = rmax; s_red[8 + wid] = rnan; s_red[16 + wid] = rinf; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0, c = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a = fmax(a, s_red[w]); b = fmax(b, s_red[8 + w]); c = fmax(c, s_red[16 + w]);
    }
    red[3 * blockIdx.x + 0] = a; red[3 * blockIdx.x + 1] = b; red[3 * blockIdx.x + 2] = c;
    __threadfence();
    unsigned done = atomicAdd(counter, 1u);
    s_last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (s_last) {   // the whole last block reduces the block maxima
    __threadfence();
    double a = 0, b = 0, c = 0;
    for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) {
      a = fmax(a, ((volatile double*)red)[3 * q]);
      b = fmax(b, ((volatile double*)red)[3 * q + 1]);
      c = fmax(c, ((volatile double*)red)[3 * q + 2]);
    }
    a = warp_max(a); b = warp_max(b); c = warp_max(c);
    __syncthreads();
    if (lane == 0) { s_red[wid] = a; s_red[8 + wid] = b; s_red[16 + wid] = c; }
    __syncthreads();
    if (threadIdx.x == 0) {
      a = 0; b = 0; c = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        a = fmax(a, s_red[w]); b = fmax(b, s_red[8 + w]); c = fmax(c, s_red[16 + w]);
      }
      double rat_max = (b > 0 || c > 0) ? 0.0 : a;  // nan_to_num(nan=0, posinf=0)
      double n = ceil(rat_max);
      int N = n > 2.0e9 ? 2000000000 : (int)n;
      if (N < 1) N = 1;
      if (N > P.max_substeps) N = P.max_substeps;
      *nsub_out = N;
      *counter = 0u;
    }
  }
}

// Per-substep component balance of PVT runs (simulation.py:1396-1505): item
// s * nwells + w replays the substeps up to s at well w's cell.  contrib[4 item + q]:
// the addend of bal[6 + {0, 1, 3, 4}[q]] (never negative), -1 where the reference
// adds nothing.
__device__ __noinline__ void well_replay(const ModelParams& P, const PvtSmem& T, const WellArgs& A, int it, int N,
                                         const double* __restrict__ p_new, double dt, double* contrib) {
  const double dt_sub = dt / N;
  const double so_r = P.so_r;
  {
    const int s = it / P.nwells, w = it % P.nwells;
    double add[4] = {-1.0, -1.0, -1.0, -1.0};   // bal[6+0], bal[6+1], bal[6+3], bal[6+4]
    const WellDev W = A.wells[w];
    const int c = W.cell;
    if (c >= 0) {
      const double* w0 = A.state + 4 * well_slot(A.wc_cells, P.nwc, c);
      double swc = w0[0], sgc = w0[1];
      const double dws = w0[2] / N, dgs = w0[3] / N;
      for (int q = 0; q <= s; ++q) {   // the cell's state after substep s (as K4b)
        swc = swc + dws;
        sgc = sgc + dgs;
        swc = tclamp(swc, P.sw_cr, 1.0 - so_r - sgc);
        sgc = tclamp(sgc, P.sg_cr, 1.0 - so_r - swc);
      }
      const double p = p_new[c];
      const PvtAt at = pvt_at(P, T, p);
      const double Bo = pvt_val(T, C_BO, at), Bw = pvt_val(T, C_BW, at), Bg = pvt_val(T, C_BG, at);
      const double Rs = pvt_val(T, C_RS, at), Rv = pvt_val(T, C_RV, at);
      const double mu_w = pvt_val(T, C_MUW, at), mu_o = pvt_val(T, C_MUO, at), mu_g = pvt_val(T, C_MUG, at);
      KR kr = relperms(P, swc, sgc);
      double mw = kr.krw / (mu_w + 1e-12), mo = kr.kro / (mu_o + 1e-12), mg = kr.krg / (mu_g + 1e-12);
      double mt = mw + mo + mg;
      double fw_ = mw / (mt + 1e-12), fg_ = mg / (mt + 1e-12), fo_ = mo / (mt + 1e-12);
      if (W.control_bhp == 0) {
        const double q_base = (W.value * P.rate_scale) / 86400.0;
        if (W.is_injector) {
          double q_sub = W.surface_rate ? q_base * (W.injected_phase == 1 ? Bg : Bw) : q_base;
          if (W.injected_phase == 1) {
            double qg_surf = fmax(q_sub, 0.0) / fmax(Bg, 1e-12) * 86400.0;
            add[2] = qg_surf * (dt_sub / 86400.0);
            add[0] = Rv * qg_surf * (dt_sub / 86400.0);
          }
        } else {
          double q_sub;
          if (W.surface_rate) {
            switch (W.surface_phase) {
              case 0: q_sub = -(q_base / fmax(fo_ / fmax(Bo, 1e-12) + fg_ * Rv / fmax(Bg, 1e-12), 1e-12)); break;
              case 1: q_sub = -(q_base * Bw) / fmax(fw_, 1e-12); break;
              case 2: q_sub = -(q_base / fmax(fg_ / fmax(Bg, 1e-12) + fo_ * Rs / fmax(Bo, 1e-12), 1e-12)); break;
              default:
                q_sub = -(q_base / fmax(fo_ / fmax(Bo, 1e-12) + fg_ * Rv / fmax(Bg, 1e-12) +
                                          fw_ / fmax(Bw, 1e-12), 1e-12));
            }
          } else {
            q_sub = -q_base;
          }
          double qo_res = fmax(-q_sub * fo_, 0.0), qg_res = fmax(-q_sub * fg_, 0.0);
          add[1] = dt_sub * (qo_res / fmax(Bo, 1e-12) + Rv * qg_res / fmax(Bg, 1e-12));
          add[3] = dt_sub * (qg_res / fmax(Bg, 1e-12) + Rs * qo_res / fmax(Bo, 1e-12));
        }
      } else {
        double q_sub = W.well_index * mt * (p - W.value * 1e6);
        if (W.is_injector) {
          if (W.injected_phase == 1) {
            double qg_surf = fmax(-q_sub, 0.0) / fmax(Bg, 1e-12) * 86400.0;
            add[2] = qg_surf * (dt_sub / 86400.0);
            add[0] = Rv * qg_surf * (dt_sub / 86400.0);
          }
        } else {
          double qabs = fabs(q_sub);
          double qo_res = qabs * fo_, qg_res = qabs * fg_;
          add[1] = dt_sub * (qo_res / fmax(Bo, 1e-12) + Rv * qg_res / fmax(Bg, 1e-12));
          add[3] = dt_sub * (qg_res / fmax(Bg, 1e-12) + Rs * qo_res / fmax(Bo, 1e-12));
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) contrib[(size_t)it * 4 + q] = add[q];
  }
}

// K4b: N clamped substeps per cell, So, and the mass balance (simulation.py:1381-1527).
constexpr int kSatBlock = 256;
__global__ void __launch_bounds__(kSatBlock, 4) k_saturation_substeps(
    ModelParams P, const double* __restrict__ pvt_g, const double* __restrict__ p_new,
    double* __restrict__ sw, double* __restrict__ sg, double* __restrict__ so,
    const double* __restrict__ dsw, const double* __restrict__ dsg, const double* __restrict__ pv,
    const int* __restrict__ nsub, double* __restrict__ red, unsigned* __restrict__ counter, WellArgs A,
    double dt, double* contrib, const int* pred) {
  double* bal = A.bal;
  if (pred && *pred == 0) return;
  __shared__ double s_col[kPvtCols * kMaxPvtRows];
  __shared__ double s_slope[(kPvtCols - 1) * kMaxPvtRows];
  __shared__ double s_w[kSatBlock / 32];
  __shared__ bool s_last;
  PvtSmem T{P.pvt_rows, s_col, s_slope};
  if (P.pvt_rows > 0) pvt_stage(pvt_g, P.pvt_rows, s_col, s_slope);
  const int N = *nsub;
  const double so_r = P.so_r;
  double acc[6] = {0, 0, 0, 0, 0, 0};  // water in/out, oil in/out, gas in/out
  const int items = P.pvt_rows > 0 ? N * P.nwells : 0;
  for (int it = dealt_first(); it < items; it += blockDim.x * gridDim.x) well_replay(P, T, A, it, N, p_new, dt, contrib);
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < P.N;
       c += (long long)gridDim.x * blockDim.x) {
    const double sw0 = sw[c], sg0 = sg[c];
    const double dws = dsw[c] / N, dgs = dsg[c] / N;
    double swc = sw0, sgc = sg0;
    for (int s = 0; s < N; ++s) {
      const double w_ = swc, g_ = sgc;
      swc = swc + dws;
      sgc = sgc + dgs;
      swc = tclamp(swc, P.sw_cr, 1.0 - so_r - sgc);
      sgc = tclamp(sgc, P.sg_cr, 1.0 - so_r - swc);
      if (swc == w_ && sgc == g_) break;   // a substep that changes nothing: nor do the others
    }
    sw[c] = swc;
    sg[c] = sgc;
    so[c] = 1.0 - swc - sgc;
    const double dwe = swc - sw0, dge = sgc - sg0;
    const double p = p_new[c], pvc = pv[c];
    // no mass moves; where a density may be NaN or infinite, zero times it is NaN
    if (dwe == 0.0 && dge == 0.0 && P.pvt_finite && isfinite(p) && isfinite(pvc)) continue;
    Rho r = densities(P, T, p, pvt_at(P, T, p));
    const double mw = dwe * pvc * r.w;
    const double mg = dge * pvc * r.g;
    const double mo = (-(dwe + dge)) * pvc * r.o;
    acc[0] += tclamp_min(mw, 0.0); acc[1] += -tclamp_max(mw, 0.0);
    acc[2] += tclamp_min(mo, 0.0); acc[3] += -tclamp_max(mo, 0.0);
    acc[4] += tclamp_min(mg, 0.0); acc[5] += -tclamp_max(mg, 0.0);
  }
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    double v = block_sum<kSatBlock>(acc[q], s_w);
    if (threadIdx.x == 0) red[6 * blockIdx.x + q] = v;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned done = atomicAdd(counter, 1u);
    s_last = (done == gridDim.x - 1);
  }
  __syncthreads();
  if (s_last) {   // the whole last block sums the block partials (fixed order)
    __threadfence();
    double tot[6] = {0, 0, 0, 0, 0, 0};
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
      for (int q = 0; q < 6; ++q) tot[q] += ((volatile double*)red)[6 * b + q];
#pragma unroll
    for (int q = 0; q < 6; ++q) tot[q] = block_sum<kSatBlock>(tot[q], s_w);
    // component balance: the wells' terms in configuration order, then the
    // replayed substeps' (warp q: oil in, oil out, gas in, gas out)
    __shared__ double s_bal[4];
    const int wq = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (wq < 4) {
      constexpr int U = 8;             // loads in flight
      double t = 0.0;
      for (int it = lane; it < items; it += 32 * U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = it + 32 * u < items ? __ldcg(contrib + 4 * (size_t)(it + 32 * u) + wq) : -1.0;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (!(v[u] < 0.0)) t += v[u];  // NaN propagates
      }
      t = warp_sum(t);
      const int bit = wq == 0 ? 8 : wq == 1 ? 16 : wq == 2 ? 32 : 64;
      double v = bal[6 + (wq < 2 ? wq : wq + 1)];
      for (int w0 = 0; w0 < P.nwells; w0 += 32) {   // 32 wells loaded at once, added one after another
        const int w = w0 + lane;
        const bool on = w < P.nwells && (A.terms[w].mask & bit);
        const double mine = on ? A.terms[w].b[wq] : 0.0;
        for (unsigned m = __ballot_sync(0xffffffffu, on); m; m &= m - 1)
          v += __shfl_sync(0xffffffffu, mine, __ffs(m) - 1);
      }
      if (lane == 0) s_bal[wq] = v + t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // mass_balance[water/oil/gas][in/out] (simulation.py:1521-1526)
      for (int q = 0; q < 6; ++q) bal[q] += tot[q];
      // component accum = in - out (simulation.py:1529-1530)
      bal[6 + 0] = s_bal[0];
      bal[6 + 1] = s_bal[1];
      bal[6 + 2] = s_bal[0] - s_bal[1];
      bal[6 + 3] = s_bal[2];
      bal[6 + 4] = s_bal[3];
      bal[6 + 5] = s_bal[2] - s_bal[3];
      *counter = 0u;
    }
  }
}

}  // namespace

// Blocks of a kernel over cells: as many as fit on the SMs at once (per_sm by its
// registers), each with several runs of cells, so that staging the PVT table and
// the block sums are paid once for them and no partial wave is left.
inline unsigned cell_grid(long long n, int per_sm) {
  return (unsigned)std::max<long long>(1, std::min<long long>((n + kCells - 1) / kCells, (long long)num_sms() * per_sm));
}

// Formation volume factors that are nowhere negative (so that the 1e-12 of the
// divisors stands above an interpolation's rounding), numbers and slopes that are
// finite and far from overflow, pressures in ascending order.
bool pvt_densities_finite(const ModelParams& P, const double* pvt) {
  const double top = 1e140;             // products and quotients by 1e-12 of such stay finite
  auto plain = [&](double v) { return v > -top && v < top; };
  if (!plain(P.rho_w_ref) || !plain(P.rho_o_ref) || !plain(P.rho_g_ref)) return false;
  for (int r = 0; r < P.pvt_rows; ++r) {
    const double* a = pvt + (size_t)r * kPvtCols;
    const double* before = r > 0 ? a - kPvtCols : nullptr;
    if (!plain(a[0]) || (before && !(a[0] > before[0]))) return false;
    for (int c : {C_BO, C_BW, C_BG, C_RS, C_RV}) {
      if (!plain(a[c]) || (before && !plain((a[c] - before[c]) / (a[0] - before[0])))) return false;
      if (c != C_RS && c != C_RV && a[c] < 0.0) return false;
    }
  }
  return true;
}

// ---------------------------------------------------------------- host API
void model_build_static(Model& m, const double* kx, const double* ky, const double* kz,
                        const double* poro, cudaStream_t s) {
  const ModelParams& P = m.P;
  m.tx.alloc(std::max<long long>(1, (long long)(P.nx - 1) * P.ny * P.nz));
  m.ty.alloc(std::max<long long>(1, (long long)P.nx * (P.ny - 1) * P.nz));
  m.tz.alloc(std::max<long long>(1, (long long)P.nx * P.ny * (P.nz - 1)));
  m.pv.alloc(P.N);
  k_transmissibility<<<grid_for(P.N, 256), 256, 0, s>>>(P, kx, ky, kz, poro, m.tx.p, m.ty.p,
                                                        m.tz.p, m.pv.p); ::impes::count_launch();
  IMPES_CHECK_LAUNCH();
  const long long faces = (long long)(P.nx - 1) * P.ny * P.nz + (long long)P.nx * (P.ny - 1) * P.nz +
                          (long long)P.nx * P.ny * (P.nz - 1);
  m.nnz = (int)(P.N + 2 * faces);
  m.rowptr.alloc(P.N + 1);
  m.col.alloc(m.nnz);
  k_pattern<<<grid_for(P.N + 1, 256), 256, 0, s>>>(P, m.nnz, m.rowptr.p, m.col.p); ::impes::count_launch();
  IMPES_CHECK_LAUNCH();
  m.red_blocks = (int)cell_grid(P.N, 4);
  m.props.alloc((size_t)5 * P.N);
  m.red.alloc((size_t)6 * m.red_blocks + 16);
  m.counter.alloc(2);
  IMPES_CUDA(cudaMemsetAsync(m.counter.p, 0, 2 * sizeof(unsigned), s));
  m.nsub.alloc(1);
  m.dsw.alloc(P.N);
  m.dsg.alloc(P.N);
  if (P.pvt_rows > 0) {
    m.pvt_tab.alloc((size_t)(2 * kPvtCols - 1) * P.pvt_rows);
    k_pvt_table<<<1, 256, 0, s>>>(P.pvt_rows, m.pvt.p, m.pvt_tab.p); ::impes::count_launch();
    IMPES_CHECK_LAUNCH();
  }
  m.wterms.alloc(std::max<size_t>(1, (sizeof(WellTerms) / sizeof(double)) * P.nwells));
  m.wstate.alloc(std::max(1, 4 * P.nwc));
  m.wsub.alloc(std::max<size_t>(1, (size_t)4 * std::max(P.max_substeps, 1) * std::max(P.nwells, 1)));
}

void model_pattern(Model& m, int* rowptr, int* col, cudaStream_t s) {
  IMPES_CUDA(cudaMemcpyAsync(rowptr, m.rowptr.p, sizeof(int) * (m.P.N + 1), cudaMemcpyDeviceToDevice, s));
  IMPES_CUDA(cudaMemcpyAsync(col, m.col.p, sizeof(int) * m.nnz, cudaMemcpyDeviceToDevice, s));
}

void model_assemble(Model& m, const double* p, const double* sw, const double* sg, double dt,
                    double* csr_val, double* rhs, cudaStream_t s) {
  const double F = 0.5 * (double)(m.nnz - m.P.N);
  const int tid = timers().begin(IMPES_PH_ASSEMBLE, s);
  const size_t n = m.P.N;
  double *mt = m.props.p, *gs = mt + n, *mo = gs + n, *pc = mo + n, *acc = pc + n;
  k_cell_props<<<cell_grid(n, 4), kCells, 0, s>>>(m.P, m.pvt_tab.p, p, sw, sg, m.pv.p, dt, mt, gs, mo, pc, acc);
  k_assemble<<<cell_grid(n, 3), kCells, 0, s>>>(m.P, p, mt, gs, mo, pc, acc, m.tx.p, m.ty.p, m.tz.p, m.wells.p, m.wc_cells.p,
                                  m.wc_ptr.p, m.wc_wells.p, m.well_mode.p, csr_val, rhs);
  ::impes::count_launches(2);
  IMPES_CHECK_LAUNCH();
  timers().end(tid, s, 8.0 * (6.0 * m.P.N + 3.0 * F));   // reads p, Sw, Sg, PV, T; writes A, b
}

void model_saturation(Model& m, const double* p_new, double* sw, double* sg, double* so, double dt,
                      cudaStream_t s, const int* pred) {
  const ModelParams& P = m.P;
  const int tid = timers().begin(IMPES_PH_SATURATION, s);
  const size_t n = P.N;
  double *mw = m.props.p, *mg = mw + n, *rw = mg + n, *rg = rw + n, *pcg = rg + n;
  const WellArgs A{m.wells.p, m.wc_cells.p, m.wc_ptr.p, m.wc_wells.p, reinterpret_cast<WellTerms*>(m.wterms.p),
                   m.wstate.p, m.balances.p, m.well_q.p, m.well_rates.p};
  k_flux_props<<<cell_grid(n, 4), kCells, 0, s>>>(P, m.pvt_tab.p, p_new, sw, sg, m.pv.p, dt, mw, mg, rw, rg, pcg, A,
                                                  pred);
  k_saturation_flux<<<cell_grid(n, 3), kCells, 0, s>>>(P, p_new, mw, mg, rw, rg, pcg, sw, sg, m.tx.p, m.ty.p, m.tz.p,
                                                       m.pv.p, A, dt, m.dsw.p, m.dsg.p, m.red.p, m.counter.p,
                                                       m.nsub.p, pred);
  k_saturation_substeps<<<cell_grid(n, 4), kSatBlock, 0, s>>>(P, m.pvt_tab.p, p_new, sw, sg, so, m.dsw.p, m.dsg.p,
                                                              m.pv.p, m.nsub.p, m.red.p, m.counter.p + 1, A, dt,
                                                              m.wsub.p, pred);
  ::impes::count_launches(3);
  IMPES_CHECK_LAUNCH();
  timers().end(tid, s, 8.0 * (6.0 * P.N + 0.5 * (double)(m.nnz - P.N)));
}

}  // namespace impes
