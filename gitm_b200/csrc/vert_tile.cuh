// vert_tile.cuh -- the Rusanov step on GITM arrays for tiles of up to
// 512 / nAlts columns: the kernel behind the 512-thread shape.
//
// What bounds a step is the latency of each phase's FP64 chains, and a
// tile's time hardly depends on how many columns it holds; so the tile takes
// every column that 512 item threads can serve (10 of 50 altitudes), and no
// phase leaves most warps waiting:
//
//  * One copy of the stage state in shared memory.  What only one thread
//    ever touches -- Orig, the RK accumulator and the stage's increments of
//    its cell, 57 doubles -- lives in tensor memory, idle otherwise without a
//    contraction on the path: 256 KB per SM, 64 doubles for each of 512 threads, written and
//    read by the thread's own warp (tcgen05.st / tcgen05.ld).  A column then
//    needs 20 KB of shared memory at 50 altitudes.  A stage is three phases:
//      P  set_vertical_bcs on every column and the limited slopes
//      B  advance_vertical_1stage at every cell, increments to tensor memory
//      C  the RK combination, each thread its own cell
//  * P is a queue of warp-sized tasks: the ions' boundaries of three columns
//    (lanes over ions), the upper boundary of two and the lower boundary of two
//    (lanes over species), each with the slopes next to its ghost cells, and
//    the slopes of 32 (field, run of about 16 cells) pairs.  The boundary chains, which kept
//    every warp busy for a fifth of the step, run beside the slopes.  A run
//    slides along its cells: one load and one difference per slope instead
//    of five and two.
//
// Each phase's code stands once in the kernel, inside the loop over stages:
// straight-line FP64 code is long (a stage is 35 KB), and the version whose
// end-of-step pass and boundaries were separate copies (249 KB instead of
// 140 KB) missed the instruction cache four times as often.
//
// Row pitches are odd, so lanes over fields of one column do not collide, and
// the column stride keeps items on consecutive banks across columns.
//
// Measured (1 degree globe, 64,800 columns of 50 altitudes, 16 steps): 59.3 ms
// with the earlier 8-column shape (Orig and accumulators in global scratch),
// 56.3 with the LDL^T friction, 48.2 with tensor memory, 10 columns and the
// task queue, 41.8 with single copies of the code and the batched exp / log,
// 38.5 with the conflict-free column stride.  Uneven ensemble (nAlts 50 / 75 /
// 100, 2 steps): 11.1 -> 7.06 ms.
#pragma once

#include "vert_kernel.cuh"
#include "vert_tmem.cuh"

namespace gv {

constexpr int TILE_THREADS = 512;
constexpr int TILE_WARPS = TILE_THREADS / 32;
constexpr int TILE_MAX_COLS = 64;              // 512 threads / 8 altitudes
constexpr int TILE_HDR = 8 + TILE_MAX_COLS;    // doubles ahead of the columns: control words, status words
constexpr int TILE_SB = 48;                    // boundary scratch of a column: lower 24, upper 24
constexpr int SC_IDFN = 60;                    // 1 / dAlt_F(nAlts)

// Tensor memory of a thread: columns (32 bits) of its 128: three blocks of 20 doubles (the 19
// fields), read as groups of 8, 8 and 4
constexpr int TM_K = 0, TM_ACC = 40, TM_O = 80;
static_assert(NF > 16 && NF <= 20, "a block holds the fields");

__host__ __device__ inline Layout make_tile_layout(int nAlts) {
  Layout L;
  L.nAlts = nAlts;
  L.G = nAlts + 4;
  L.P = L.G | 1;
  L.PD = (nAlts + 2) | 1;
  L.nsl = NSTENCIL;
  int o = 0;
  L.X0 = o;  o += NF * L.P;
  L.XP0 = o; o += NPAS * NPC;
  L.X1 = L.X0;
  L.XP1 = L.XP0;
  L.O = L.OP = L.LT = 0;
  L.OGH = o; o += NADV * 2 + NPAS * NPC;
  L.DL = o;  o += NSTENCIL * L.PD;
  L.TU = o;  o += L.G;
  L.CM = o;  o += L.G;
  L.GM = o;  o += L.G;
  L.SC = o;  o += NSC;
  L.QS = o;  o += TILE_SB;
  // items of neighbouring columns fall on neighbouring banks (16 of a double):
  // item t of every row is at t modulo 16
  while (o % 16 != nAlts % 16) ++o;
  L.stride = o;
  return L;
}

__host__ __device__ inline size_t tile_smem_bytes(int nAlts, int nc) {
  return (size_t(make_tile_layout(nAlts).stride) * nc + TILE_HDR) * sizeof(double);
}

// ------------------------------------------------------------ slopes
// The limited slope of field f at any cell 0..nAlts+1 (rusanov_slopes_cell
// for one field): the cells next to the ghosts.
__device__ __forceinline__ void tile_slope(const ColCtx& c, int f, int i, double beta) {
  const int nA = c.L.nAlts;
  const bool end = (i == 0 || i == nA + 1);
  const double cu = end ? c.g(GC_IDF, i + 1) : c.g(GC_H2, i + 1);
  const double cd = end ? c.g(GC_IDF, i) : c.g(GC_H2, i);
  const double a = end ? 1.0 : F1, b = end ? 0.0 : F2;
  const int ip2 = min(i + 2, nA + 2), im2 = max(i - 2, -1);
  const double* v = c.col + c.xo + 1 + f * c.L.P;
  const double u = cu * (a * (v[i + 1] - v[i]) - b * (v[ip2] - v[i - 1]));
  const double d = cd * (a * (v[i] - v[i - 1]) - b * (v[i + 1] - v[im2]));
  c.dl(f, i) = limiter_mc(u, d, beta);
}

// Slopes of field f at cells i0 .. i1-1 (within 3 .. nAlts-2: interior
// neighbours only), sliding along the row.
__device__ __forceinline__ void tile_slope_run(const ColCtx& c, int f, int i0, int i1, double beta) {
  const double* __restrict__ v = c.col + c.xo + 1 + f * c.L.P;
  double* __restrict__ sl = c.col + c.L.DL + f * c.L.PD;
  double vm = v[i0 - 1], v0 = v[i0], vp = v[i0 + 1];
  double d = c.g(GC_H2, i0) * (F1 * (v0 - vm) - F2 * (vp - v[i0 - 2]));
#pragma unroll 4
  for (int i = i0; i < i1; ++i) {
    const double vq = v[i + 2];
    const double u = c.g(GC_H2, i + 1) * (F1 * (vp - v0) - F2 * (vq - vm));
    sl[i] = limiter_mc(u, d, beta);
    d = u;
    vm = v0;
    v0 = vp;
    vp = vq;
  }
}

// ------------------------------------------------------------ boundaries
// set_vertical_bcs (set_vertical_bcs.Earth.f90:8-652) as bc_column forms it,
// split over groups of lanes so that a warp serves several columns.  The
// lower boundary, by six lanes per column (s = species):
__device__ __forceinline__ void tile_lower(const ColCtx& c, const GitmVertParams& prm, bool act, int s) {
  double* X = c.col + c.xo + 1;
  const int P = c.L.P;
  const double* sc = c.col + c.L.SC;
  double* sb = c.col + c.L.QS;
  auto x = [&](int f, int i) -> double& { return X[f * P + i]; };
  const bool msis = prm.use_msis_bcs && sc[SC_HASLBC] != 0.0;
  const double* bl = sc + SC_BCC;  // mesh coefficients, cell 0 then -1
  if (act) {
    // lines 112-148, 192-196 (Temp, Vel_GD: one lane each)
    const double* t = sc + SC_LBC;
    const double l0 = x(F_LNS + s, 0);  // NS(0) of line 93, before the MSIS values
    const double T0 = msis ? t[16] : x(F_T, 0);
    if (s == 0) {
      x(F_T, 0) = T0;
      x(F_T, -1) = T0;
    } else if (s == 1 || s == 2) {
      const int f = (s == 1) ? F_VE : F_VN;
      const double v = msis ? t[17 + s] : 0.0;
      x(f, 0) = v;
      x(f, -1) = v;
    }
    double n0 = msis ? t[10 + s] : l0, n1;
    if (!photochemical(s)) {
      // lines 205-222: hydrostatic cell -1 with the mean major mass
      const double MeanGravity = -0.5 * (sc[SC_EG + 0] + sc[SC_EG + 1]);
      const double MeanTemp = 0.5 * (T0 + T0);
      const double MeanMass = 0.5 * (sc[SC_MMM_0] + sc[SC_MMM_M1]);
      const double ish = MeanGravity * MeanMass / (MeanTemp * KB);
      n1 = (s == 0) ? n0 : l0 + ish * sc[SC_DAF + 0];
    } else {
      // lines 226-272: 3rd-order extrapolation with a gradient limit
      double p[6];  // cells 0 (set first) .. 5
#pragma unroll
      for (int q = 1; q < 6; ++q) p[q] = x(F_LNS + s, q);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const double* C = bl + 5 * k;
        const double up = p[1 - k];
        double d;
        if (k == 0)
          d = p[1] * C[0] + p[2] * C[1] + p[3] * C[2] + p[4] * C[3] + p[5] * C[4];
        else
          d = p[0] * C[0] + p[1] * C[1] + p[2] * C[2] + p[3] * C[3] + p[4] * C[4];
        double v = up - sc[SC_DAF + 2 - k] * d;
        if (d <= 0.0) v = up;
        if (s == 4 && v < up - 0.333) v = up - 0.333;
        if (k == 0)
          p[0] = v;
        else
          n1 = v;
      }
      n0 = p[0];
    }
    x(F_LNS + s, 0) = n0;
    x(F_LNS + s, -1) = n1;
    // vertical winds (lines 334-344)
    const double w1 = x(F_W + s, 1);
    double w0 = w1 - sc[SC_DAF + 2] * (w1 * bl[0] + x(F_W + s, 2) * bl[1] + x(F_W + s, 3) * bl[2] +
                                       x(F_W + s, 4) * bl[3] + x(F_W + s, 5) * bl[4]);
    double wm = w0 - sc[SC_DAF + 1] * (w0 * bl[5] + w1 * bl[6] + x(F_W + s, 2) * bl[7] + x(F_W + s, 3) * bl[8] +
                                       x(F_W + s, 4) * bl[9]);
    const double l[2] = {n0, n1};
    double e[2];
    exp_n(l, e);
    const double m0 = c_k.mass[s] * e[0];
    const double m1 = c_k.mass[s] * e[1];
    sb[s] = m0;
    sb[NS + s] = m1;
    sb[2 * NS + s] = m0 * w0;
    sb[3 * NS + s] = m1 * wm;
    // lines 382-395
    if (photochemical(s) && w1 > 0.0) {
      w0 = -1.0 * w1;
      wm = -1.0 * w1;
    }
    x(F_W + s, 0) = w0;
    x(F_W + s, -1) = wm;
  }
  __syncwarp();
  if (act) {
    // lines 348-362: LogRho and the bulk vertical wind at cells 0 and -1
    if (s < 2) {
      double r = 0.0, v = 0.0;
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        r = r + sb[s * NS + k];
        v = v + sb[(2 + s) * NS + k];
      }
      x(F_LRHO, -s) = log_sl(r);
      x(F_VU, -s) = v / r;
    } else if (msis && s < 4) {
      // lines 364-376
      const int f = (s == 2) ? F_VE : F_VN;
      const double* C = bl + 5;
      const double d = x(f, 0) * C[0] + x(f, 1) * C[1] + x(f, 2) * C[2] + x(f, 3) * C[3] + x(f, 4) * C[4];
      x(f, -1) = x(f, 0) - sc[SC_DAF + 1] * d;
    }
  }
  __syncwarp();
}

// The upper boundary's winds, temperature and neutral densities, by six lanes
// per column.
__device__ __forceinline__ void tile_upper(const ColCtx& c, bool act, int s) {
  const int nA = c.L.nAlts;
  double* X = c.col + c.xo + 1;
  const int P = c.L.P;
  const double* sc = c.col + c.L.SC;
  double* sb = c.col + c.L.QS + 24;
  auto x = [&](int f, int i) -> double& { return X[f * P + i]; };
  if (act) {
    // lines 434-454: species winds; 471-486: hydrostatic densities
    const double wn = x(F_W + s, nA);
    double w1 = wn, w2 = wn;
    if (photochemical(s) && wn < 0.0) {
      w1 = -wn;
      w2 = -x(F_W + s, nA - 1);
    }
    x(F_W + s, nA + 1) = w1;
    x(F_W + s, nA + 2) = w2;
    const double T = x(F_T, nA);
    const double mr = c_k.mass[s] * rcp_nr(0.5 * (T + T) * KB);
    const double ish1 = (-0.5 * (sc[SC_EG + 3] + sc[SC_EG + 2])) * mr;
    const double ish2 = (-0.5 * (sc[SC_EG + 4] + sc[SC_EG + 3])) * mr;
    const double l1 = x(F_LNS + s, nA) - ish1 * sc[SC_DAF + 4];
    const double l2 = l1 - ish2 * sc[SC_DAF + 5];
    x(F_LNS + s, nA + 1) = l1;
    x(F_LNS + s, nA + 2) = l2;
    const double l[2] = {l1, l2};
    double e[2];
    exp_n(l, e);
    sb[s] = c_k.mass[s] * e[0];
    sb[NS + s] = c_k.mass[s] * e[1];
    // lines 420-430, 455-469, a field per lane
    if (s < 4) {
      const int f = F_T + s;  // Temp, Vel_GD east, north, up
      double v = x(f, nA);
      if (f == F_VU) v = fabs(v);
      x(f, nA + 1) = v;
      x(f, nA + 2) = v;
    }
  }
  __syncwarp();
  // lines 598-604
  if (act && s < 2) {
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) r = r + sb[s * NS + k];
    x(F_LRHO, nA + 1 + s) = log_sl(r);
  }
  __syncwarp();
}

// Both boundaries' ions, by nine lanes per column (s = ion); first: the
// group's lane 0.  Returns true where the negative-density repair changed
// interior cells.
__device__ __forceinline__ bool tile_ions(const ColCtx& c, const GitmVertParams& prm, bool act, int s, int first,
                                                uint32_t* st) {
  constexpr unsigned ALL = 0xffffffffu;
  const int nA = c.L.nAlts;
  const double* sc = c.col + c.L.SC;
  double* sb = c.col + c.L.QS + 36;
  const bool improved = prm.use_improved_ion_advection != 0;
  double n[7];  // ion s at cells nAlts+2, nAlts+1, .., nAlts-4
  bool neg = false;
#pragma unroll
  for (int j = 0; j < 7; ++j) n[j] = 1.0;
  if (act) {
#pragma unroll
    for (int j = 0; j < 7; ++j) n[j] = c.ion(s, nA + 2 - j);
    if (improved) {
#pragma unroll
      for (int j = 0; j < 7; ++j) neg = neg || n[j] < 0.0;
      neg = neg || c.ion(s, nA - 5) < 0.0;
    }
    // ions float at the lower boundary (lines 304-310)
    const double v = c.ion(s, 1);
    c.ion(s, 0) = v;
    c.ion(s, -1) = v;
  }
  bool hold = false;
  const bool night = act && sc[SC_PLASMA] != 0.0;
  if (__any_sync(ALL, night)) {
    // lines 488-501: the TEC of the first ion, needed where the plasma switch is on
    if (night) {
      double tp = 0.0;
      for (int i = 1 + s; i <= nA; i += NI) tp += c.dAF(i) * (improved ? c.ion(0, i) : exp_sl(c.ion(0, i)));
      sb[s] = tp;
    }
    __syncwarp();
    if (night) {
      double tp = 0.0;
#pragma unroll
      for (int k = 0; k < NI; ++k) tp += sb[k];
      hold = tp < prm.min_tec * 1e16;  // TEC / 1e16 < MinTEC
    }
    __syncwarp();
  }
  const bool anyneg = ((__ballot_sync(ALL, act && neg) >> first) & 0x1ffu) != 0u;
  // lines 503-649
  const double* C = sc + SC_BCC + 10;  // mesh coefficients, nAlts+1 then nAlts+2
  const double* D = C + 5;
  double v1 = 0.0, v2 = 0.0;
  {
    // without negative values; with UseImprovedIonAdvection on the logs
    double m[7];
    if (improved)
      log_n(n, m);
    else
#pragma unroll
      for (int j = 0; j < 7; ++j) m[j] = n[j];
    double dn = C[0] * m[2] + C[1] * m[3] + C[2] * m[4] + C[3] * m[5] + C[4] * m[6];
    const double lim = -(0.001 * m[1] * sc[SC_IDFN]);
    if (dn > lim) dn = lim;
    v1 = m[2] + dn * sc[SC_DAF + 4];
    // cell nAlts+2: the value just set stands for its own log
    double dn2 = D[0] * v1 + D[1] * m[2] + D[2] * m[3] + D[3] * m[4] + D[4] * m[5];
    const double lim2 = -(0.001 * m[0] * sc[SC_IDFN]);
    if (dn2 > lim2) dn2 = lim2;
    v2 = v1 + dn2 * sc[SC_DAF + 5];
    if (improved) {
      const double y[2] = {v1, v2};
      double e[2];
      exp_n(y, e);
      v1 = e[0];
      v2 = e[1];
    }
  }
  if (act) {
    if (!anyneg) {
      if (!hold) {
        c.ion(s, nA + 1) = v1;
        c.ion(s, nA + 2) = v2;
      }
    } else {
      // the reference's order, one ion per lane
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        const int iAlt = nA + 1 + k;
        double mn = c.ion(s, iAlt - 5);
        for (int q = iAlt - 4; q <= iAlt; ++q) mn = fmin(mn, c.ion(s, q));
        if (mn < 0.0) {
          if (c.ion(s, iAlt - 6) < 0.0) atomicOr(st, GITM_ST_NEG_ION_TOP);
          for (int q = iAlt - 5; q <= iAlt - 1; ++q) {
            if (c.ion(s, q) < 0.0) {
              if (c.ion(s, q - 1) > 0.0 && c.ion(s, q + 1) > 0.0)
                c.ion(s, q) = (c.ion(s, q - 1) + c.ion(s, q + 1)) / 2.0;
              else
                c.ion(s, q) = c.ion(s, q - 1) * 0.95;
            }
          }
          if (c.ion(s, iAlt) < 0.0) c.ion(s, iAlt) = c.ion(s, iAlt - 1) * 0.95;
        }
        if (!hold) {
          double dn = 0.0;
          for (int j = 1; j < 6; ++j) dn = dn + C[5 * k + j - 1] * log_sl(c.ion(s, iAlt - j));
          const double lim = -(0.001 * log_sl(c.ion(s, iAlt)) / sc[SC_DAF + 3]);
          if (dn > lim) dn = lim;
          c.ion(s, iAlt) = exp_sl(log_sl(c.ion(s, iAlt - 1)) + dn * sc[SC_DAF + 4 + k]);
        }
      }
    }
  }
  __syncwarp();
  return act && anyneg;
}

// Gamma, MeanMajorMass, TempUnit and the cell's cMax (calc_pressure.f90:17-21,
// 56-83; calc_rates.Earth.f90:34-50; calc_timestep.f90:114-118).
__device__ __forceinline__ void tile_producers(const double (&nd)[NS], const double (&ww)[NS], double temperature,
                                               double& gamma, double& mmm, double& tu, double& cmx) {
  double N = 0.0, gg = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    N = N + nd[s];
    gg = gg + nd[s] * c_k.inv_vib2[s];
  }
  gamma = gg * 2.0 / N + 1;
  double m = 0.0;
  const double rn = 1.0 / (N + 1.0);
#pragma unroll
  for (int s = 0; s < NS; ++s) m = m + c_k.mass[s] * nd[s] * rn;
  if (m == 0) m = c_k.mass[0];
  mmm = m;
  tu = m * (1.0 / KB);
  double mx = fabs(ww[0]);
#pragma unroll
  for (int s = 1; s < NS; ++s) mx = fmax(mx, fabs(ww[s]));
  cmx = mx + sqrt(gamma * temperature);
}

// Fields F0 .. F0+N-1 of the RK combination at the thread's cell after stage
// k: see phase C.  Whole warps call it; the state is written where `item`.
template <int F0, int N>
__device__ __forceinline__ void tile_combine(const ColCtx& c, uint32_t tm, int i, bool item, int k, double ca,
                                             double cx) {
  double kv[N], a[N], o[N];
  if (k == 0) {
    // the state the stage read is Orig
    tm_get(tm + TM_K + 2 * F0, kv);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      a[j] = 0.0;
      o[j] = (F0 + j < NF) ? c.x(F0 + j, i) : 0.0;
    }
    tm_put(tm + TM_O + 2 * F0, o);
  } else {
    tm_get(tm + TM_K + 2 * F0, tm + TM_ACC + 2 * F0, tm + TM_O + 2 * F0, kv, a, o);
  }
#pragma unroll
  for (int j = 0; j < N; ++j) a[j] = fma(ca, kv[j], a[j]);
  if (k < 3) tm_put(tm + TM_ACC + 2 * F0, a);
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (F0 + j < NF && item) c.x(F0 + j, i) = o[j] + cx * ((k == 3) ? a[j] : kv[j]);
}

// add_sources' temperature line with EuvHeating its only term
// (add_sources.f90:53-66), applied after every step.
__device__ __forceinline__ double tile_heated(const GitmColumnBatch& b, double temperature, double dt, int64_t cell,
                                              int64_t col) {
  const double hs = b.heating_scale ? b.heating_scale[col] : 1.0;
  return temperature + dt * (hs * b.heating[cell]);
}

// ------------------------------------------------------------ the kernel
// kp.scratch is not used.  SAVE: see KParams::save.
template <int NA, bool SAVE>
__global__ void __launch_bounds__(TILE_THREADS, 1) vert_tile_kernel(const KParams kp) {
  extern __shared__ double sm[];
  constexpr unsigned ALL = 0xffffffffu;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int wid = tid >> 5;
  const GitmVertParams& prm = kp.prm;
  const double dt = kp.dt;
  const double inv_vert_tau = 1.0 / prm.vert_tau;
  uint32_t* ctl = reinterpret_cast<uint32_t*>(sm);  // 0: tensor-memory base; the next task of phase P (1)
                                                      // and of a step's end (3); 2: a repair changed ions
  uint32_t* sst = reinterpret_cast<uint32_t*>(sm + 8);
  uint32_t* sfrozen = sst + TILE_MAX_COLS;
  double* const cols = sm + TILE_HDR;

  if (wid == 0) tm_alloc<512>(ctl);
  if (tid == 0) {
    ctl[1] = TILE_WARPS;
    ctl[2] = 0;
    ctl[3] = TILE_WARPS;
  }
  __syncthreads();
  const uint32_t tm_base = *reinterpret_cast<volatile uint32_t*>(ctl);
  // warp w reaches the 32 lanes of its quarter; its columns by warpgroup
  const uint32_t tm = tm_base + (uint32_t(wid & 3) << 21) + uint32_t(wid >> 2) * 128u;

  for (int tix = blockIdx.x; tix < kp.n_tiles; tix += gridDim.x) {
    const Tile tile = kp.tiles[tix];
    const DevMember& M = kp.members[tile.member];
    const GitmColumnBatch& b = M.b;
    const int nA = (NA > 0) ? NA : M.b.n_alts;
    const int nc = tile.nc;
    const Layout L = make_tile_layout(nA);
    const int G = L.G;
    const int64_t ncols = M.b.n_cols;
    const int nitems = nc * nA;
    const bool item = tid < nitems;
    const bool wact = wid * 32 < nitems;  // warps with items run whole: the idle lanes of the last repeat its last item
    const int it = min(tid, nitems - 1);
    const int my_cl = it / nA;
    const int my_i = it % nA + 1;

    auto ctx = [&](int cl) {
      ColCtx c;
      c.col = cols + size_t(L.stride) * cl;
      c.L = L;
      c.gridc = M.gridc;
      c.gcols = M.gcols;
      c.gc = (M.gcols == 1) ? 0 : int(tile.c0 + cl);
      c.xo = L.X0;
      c.xpo = L.XP0;
      return c;
    };
    auto gidx = [&](int f, int g, int cl) -> int64_t { return (int64_t(f) * G + g) * ncols + tile.c0 + cl; };
    auto save_state = [&](int s) {
      if constexpr (SAVE) {
        const int per = NF * G + NPAS * NPC;
        for (int w = tid; w < nc * per; w += TILE_THREADS) {
          const int cl = w / per, r = w - cl * per;
          const int f = r / G;
          const double* col = cols + size_t(L.stride) * cl;
          const double v = (f < NF) ? col[L.X0 + f * L.P + (r - f * G)] : col[L.XP0 + r - NF * G];
          kp.save[(int64_t(s) * kp.save_ncols + M.col_offset + tile.c0 + cl - kp.save_c0) * kp.save_per + r] = v;
        }
      }
    };
    const bool dry = SAVE && kp.no_store != 0;
    // MeanMajorMass of the last step, where it is formed (only its TempUnit is kept)
    auto put_mmm = [&](int g, int cl, double mmm) {
      if (b.mean_major_mass && !dry) b.mean_major_mass[gidx(0, g, cl)] = mmm;
    };
    // the tasks of phase P
    const int ninner = nA - 4;  // cells 3 .. nAlts-2
    const int nrun = max(1, (ninner + 8) / 16);
    const int runlen = (ninner + nrun - 1) / nrun;
    const int nslope = nrun * nc * NSTENCIL;
    const int n_ion = (nc + 2) / 3, n_two = (nc + 1) / 2;  // boundary tasks: ions; upper, and lower
    const int nbc = n_ion + 2 * n_two;

    if (tid < nc) {
      sst[tid] = 0u;
      sfrozen[tid] = 0u;
    }
    __syncthreads();

    // ---------------------------------------------------------- load
    // per-column scalars (advance_vertical.f90:84-85,103-104)
    if (tid < nc) {
      ColCtx c = ctx(tid);
      const int64_t cc = tile.c0 + tid;
      const double cl = b.cos_lat[cc];
      const double cent = (cl * prm.omega_body) * (cl * prm.omega_body);
      const double sza = b.sza[cc], mlat = b.mlat[cc];
      c.sc(SC_CENT) = cent;
      c.sc(SC_CORI) = 2 * cl * prm.omega_body;
      c.sc(SC_SZA) = sza;
      c.sc(SC_MLAT) = mlat;
      // set_vertical_bcs.Earth.f90:488-495
      bool plasma = false;
      if (prm.use_nighttime_ion_bcs)
        plasma = sza > PI / 2 && ((mlat > 30.0 && mlat < 70.0) || (mlat > -60.0 && mlat < -30.0));
      c.sc(SC_PLASMA) = plasma ? 1.0 : 0.0;
      c.sc(SC_HASLBC) = b.lbc ? 1.0 : 0.0;
      if (b.lbc)
        for (int k = 0; k < 2 * GITM_LBC_NVALUES; ++k) c.sc(SC_LBC + k) = b.lbc[int64_t(k) * ncols + cc];
      for (int j = 0; j < 20; ++j) c.sc(SC_BCC + j) = c.bcc(j);
      const int dcell[6] = {-1, 0, 1, nA, nA + 1, nA + 2};
      for (int j = 0; j < 6; ++j) c.sc(SC_DAF + j) = c.dAF(dcell[j]);
      const int ecell[5] = {-1, 0, nA, nA + 1, nA + 2};
      for (int j = 0; j < 5; ++j) c.sc(SC_EG + j) = c.g(GC_GRAV, ecell[j]) + cent * c.g(GC_R, ecell[j]);
      c.sc(SC_IDFN) = c.g(GC_IDF, nA);
    }
    // columns vary fastest across threads so that a warp reads whole row
    // segments of the native layout
    for (int w = tid; w < nc * G; w += TILE_THREADS) {
      const int g = w / nc, cl = w - g * nc, i = g - 1;
      ColCtx c = ctx(cl);
      double nd[NS], ww[NS];
      double mn = 1.0;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        nd[s] = b.ndensity_s[gidx(s, g, cl)];
        ww[s] = b.vert_vel[gidx(s, g, cl)];
        mn = fmin(mn, nd[s]);
      }
      if (!(mn > 0.0)) atomicOr(&sfrozen[cl], 1u);
      const double temperature = b.temperature[gidx(0, g, cl)];
      double gamma, mmm, tu, cmx = 0.0;
      if (prm.compute_coefficients) {
        // calc_pressure.f90:17-21,56-83; calc_rates.Earth.f90:34-50; calc_timestep.f90:114-118
        tile_producers(nd, ww, temperature, gamma, mmm, tu, cmx);
        if (!(g >= 1 && g <= nA + 2)) cmx = 0.0;
        if (kp.n_steps == 1) put_mmm(g, cl, mmm);
      } else {
        gamma = b.gamma[gidx(0, g, cl)];
        mmm = b.mean_major_mass[gidx(0, g, cl)];
        tu = b.temp_unit[gidx(0, g, cl)];
        if (g >= 1 && g <= nA + 2) cmx = b.cmax[gidx(0, g, cl)];
      }
      c.tu(i) = tu;
      c.cm(i) = cmx;
      c.gm(i) = gamma;
      if (i == -1) c.sc(SC_MMM_M1) = mmm;
      if (i == 0) c.sc(SC_MMM_0) = mmm;
      double r7[NS + 1], l7[NS + 1];
#pragma unroll
      for (int s = 0; s < NS; ++s) r7[s] = nd[s];
      r7[NS] = b.rho[gidx(0, g, cl)];
      log_n(r7, l7);
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        c.x(F_LNS + s, i) = l7[s];
        c.x(F_W + s, i) = ww[s];
      }
      c.x(F_T, i) = temperature * tu;
      c.x(F_VE, i) = b.velocity[gidx(0, g, cl)];
      c.x(F_VN, i) = b.velocity[gidx(1, g, cl)];
      c.x(F_VU, i) = b.velocity[gidx(2, g, cl)];
      c.x(F_LRHO, i) = l7[NS];
      const bool pc = in_pcells(i, nA);
#pragma unroll 3
      for (int s = 0; s < NI; ++s) {
        if (s >= NADV && !pc) continue;
        const double v = b.idensity_s[gidx(s, g, cl)];
        c.ion(s, i) = prm.use_improved_ion_advection ? v : log_sl(v);
      }
    }
    __syncthreads();
    if constexpr (SAVE) {
      save_state(0);
      __syncthreads();  // the boundary pass rewrites what was just saved
    }

#pragma unroll 1
    for (int step = 0; step < kp.n_steps; ++step) {
      const double eddy = b.eddy[gidx(0, my_i + 1, my_cl)];
      const double ivup = b.ivel_up[gidx(0, my_i + 1, my_cl)];

      const bool last = (step == kp.n_steps - 1);
#pragma unroll 1
      for (int k = 0;; ++k) {
        // -------------------------------------------------- phase P
        // the boundaries (set_vertical_bcs, :95,166,236,306,368) and beside
        // them the slopes, or after the last stage (k = 4) the next step's
        // gather.  Tasks 0 .. 15 go to the warps of that number, the rest
        // from a queue.
        const bool slopes = k < 4;
        const int n_all = nbc + ((slopes ? nslope : last ? 0 : nitems) + 31) / 32;
        for (int t = wid; t < n_all;) {
          int rcl = -1, ri = 0;  // the cell whose gather this lane takes
          if (t < nbc) {
            const bool ions = t < n_ion, up = t < n_ion + n_two;
            const int q = ions ? lane / NI : lane / NS, s = ions ? lane % NI : lane % NS;
            const int cl0 = ions ? 3 * t : 2 * (up ? t - n_ion : t - n_ion - n_two);
            const int n = min(ions ? 3 : 2, nc - cl0);  // columns of this task
            const bool act = q < n;
            const int cl = act ? cl0 + q : cl0;
            if (ions) {
              if (tile_ions(ctx(cl), prm, act, s, q * NI, &sst[cl])) ctl[2] = 1;
            } else if (up) {
              tile_upper(ctx(cl), act, s);
            } else {
              tile_lower(ctx(cl), prm, act, s);
            }
            if (slopes) {
              // the slopes that reach the ghost cells set here: cells 0, 1, 2 and nAlts-1, nAlts, nAlts+1
              // (lanes over the 16 other fields of two columns, or both ends of the ions of three)
              const int c2 = lane >> (ions ? 2 : 4), fr = lane & (ions ? 3 : 15);
              static_assert(NADV == 2 && F_I == 16, "the lanes of the slopes at the ends");
              if (c2 < n) {
                ColCtx c = ctx(cl0 + c2);
                const int f = ions ? F_I + (fr & 1) : fr, e0 = (ions ? fr >= 2 : up) ? nA - 1 : 0;
#pragma unroll
                for (int e = 0; e < 3; ++e) tile_slope(c, f, e0 + e, prm.beta_limiter);
              }
            } else if (!last) {
              if (ions) {
                // the floor of every interior ion held here (the boundary above
                // read them): advected ions at cells 1 .. nAlts, passive ones at
                // 1 and nAlts-5 .. nAlts
                if (prm.use_ion_advection && prm.use_improved_ion_advection) {
                  const int na = NADV * nA, per = na + NPAS * 7;
                  for (int w = lane; w < n * per; w += 32) {
                    const int c2 = w / per, r = w - c2 * per, h = r - na;
                    const int s2 = h < 0 ? r / nA : NADV + h / 7;
                    const int i = h < 0 ? r % nA + 1 : (h % 7 == 0 ? 1 : nA - 6 + h % 7);
                    double& v = ctx(cl0 + c2).ion(s2, i);
                    if (v < 1) v = 1.0;
                  }
                }
              } else if (lane < n * 3) {
                const int c2 = lane / 3, r = lane - c2 * 3;
                if (up || r < 2) {  // the upper boundary reads Temp(nAlts): its gather comes after
                  rcl = cl0 + c2;
                  ri = up ? nA + r : -r;
                }
              }
            }
          } else {
            const int w = (t - nbc) * 32 + lane;
            if (slopes) {
              if (w < nslope) {
                const int r = w / (nc * NSTENCIL), q = w - r * (nc * NSTENCIL);
                const int cl = q / NSTENCIL, f = q - cl * NSTENCIL;
                const int i0 = 3 + r * runlen;
                tile_slope_run(ctx(cl), f, i0, min(i0 + runlen, nA - 1), prm.beta_limiter);
              }
            } else if (w < nitems) {
              ri = w / nc + 1;  // columns fastest, as in the load
              if (ri < nA) rcl = w - (ri - 1) * nc;
            }
          }
          if (rcl >= 0) {
            // LogNS and LogRho of the next gather (advance_vertical.f90:105,114)
            // are the values in X up to a rounding of exp / log: X keeps them
            ColCtx c = ctx(rcl);
            double temperature = c.x(F_T, ri) / c.tu(ri);
            if (b.heating && ri >= 1 && ri <= nA)
              temperature = tile_heated(b, temperature, dt, gidx(0, ri + 1, rcl), tile.c0 + rcl);
            double l[NS], nd[NS], ww[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
              l[s] = c.x(F_LNS + s, ri);
              ww[s] = c.x(F_W + s, ri);
            }
            exp_n(l, nd);
            bool bad = false;
#pragma unroll
            for (int s = 0; s < NS; ++s) bad = bad || !(nd[s] > 0.0);
            if (bad) atomicOr(&sst[rcl], GITM_ST_NEG_DENSITY);
            double tu = c.tu(ri);
            if (prm.compute_coefficients) {
              double gamma, mmm, cmx;
              tile_producers(nd, ww, temperature, gamma, mmm, tu, cmx);
              c.gm(ri) = gamma;
              c.cm(ri) = (ri >= 0 && ri <= nA + 1) ? cmx : 0.0;
              c.tu(ri) = tu;
              if (step == kp.n_steps - 2) put_mmm(ri + 1, rcl, mmm);
              if (ri == -1) c.sc(SC_MMM_M1) = mmm;
              if (ri == 0) c.sc(SC_MMM_0) = mmm;
            }
            c.x(F_T, ri) = temperature * tu;
          }
          if (lane == 0) t = int(atomicAdd(&ctl[slopes ? 1 : 3], 1u));
          t = __shfl_sync(ALL, t, 0);
        }
        __syncthreads();
        save_state(1 + k);
        if (!slopes) break;
        if (ctl[2] != 0) {
          // a repair changed ion cells the slope tasks may have read before it
          for (int w = tid; w < nc * NADV * 8; w += TILE_THREADS) {
            const int cl = w / (NADV * 8), r = w - cl * (NADV * 8);
            tile_slope(ctx(cl), F_I + (r >> 3), nA + 1 - (r & 7), prm.beta_limiter);
          }
          __syncthreads();
        }
        if (tid == 0) {
          ctl[1] = TILE_WARPS;
          ctl[3] = TILE_WARPS;
        }

        // -------------------------------------------------- phase B
        // advance_vertical_1stage (:387-686) at the item's cell; its
        // increments go to tensor memory
        if (wact) {
          rusanov_cell<true>(ctx(my_cl), my_i, prm, dt, eddy, ivup, inv_vert_tau,
                       [&](int f, double kval) { tm_put(tm + TM_K + 2 * f, kval); }, &sst[my_cl]);
          tm_put_wait();
        }
        __syncthreads();

        // -------------------------------------------------- phase C
        // (vertical_solver_rusanov.f90:120-163,190-232,261-303,350-366): the
        // accumulator a = prev + ca K (ca = 1, 2, 2, 1), the next state Orig
        // + cx K for k < 3 (cx = 1/2, 1/2, 1) and Orig + a / 6 after the
        // last stage; a multiplication by 1 or 2 is exact
        if (tid == 0) ctl[2] = 0;
        const double ca = (k == 1 || k == 2) ? 2.0 : 1.0;
        const double cx = (k < 2) ? 0.5 : (k == 2) ? 1.0 : 1.0 / 6.0;
        if (wact) {
          ColCtx c = ctx(my_cl);
          if (k == 0 && prm.compute_eddy && item && sfrozen[my_cl] == 0u) {
            // calc_eddy_diffusion_coefficient (Earth.f90:376-411) on Pressure =
            // Temperature * Rho (calc_pressure.f90:23) of the state this step
            // started from: the coefficient the next step reads
            const double pr = (c.x(F_T, my_i) / c.tu(my_i)) * exp_sl(c.x(F_LRHO, my_i));
            double kz = 0.0;
            if (pr > prm.eddy_pressure0)
              kz = prm.eddy_coef;
            else if (pr > prm.eddy_pressure1)
              kz = prm.eddy_coef * (pr - prm.eddy_pressure1) / (prm.eddy_pressure0 - prm.eddy_pressure1);
            b.eddy[gidx(0, my_i + 1, my_cl)] = kz;
          }
          __syncwarp();
          tile_combine<0, 8>(c, tm, my_i, item, k, ca, cx);
          tile_combine<8, 8>(c, tm, my_i, item, k, ca, cx);
          tile_combine<16, 4>(c, tm, my_i, item, k, ca, cx);
          tm_put_wait();
        }
        // what the next boundary pass reads before it sets it, the advected
        // ions' upper ghost cells and the passive ions: kept after the first
        // pass, back to that (their K is zero) after every stage.  The other
        // ghost cells it reads are LogNS(0) and Temp(0), which it leaves alone.
        {
          constexpr int per = NADV * 2 + NPAS * NPC;
          for (int w = tid; w < nc * per; w += TILE_THREADS) {
            const int cl = w / per, r = w - cl * per;
            double* col = cols + size_t(L.stride) * cl;
            double* now = col + (r < NADV * 2 ? L.X0 + (F_I + (r >> 1)) * L.P + nA + 2 + (r & 1)  // nAlts+1, nAlts+2
                                              : L.XP0 + r - NADV * 2);
            if (k == 0)
              col[L.OGH + r] = *now;
            else
              *now = col[L.OGH + r];
          }
        }
        __syncthreads();
      }
    }

    // ---------------------------------------------------------- store
    // scatter, advance_vertical.f90:163-217
    for (int w = tid; w < nc * G && !dry; w += TILE_THREADS) {
      const int g = w / nc, cl = w - g * nc, i = g - 1;
      ColCtx c = ctx(cl);
      if (prm.compute_coefficients) {
        // the coefficients the last step ran with
        if (b.gamma) b.gamma[gidx(0, g, cl)] = c.gm(i);
        if (b.temp_unit) b.temp_unit[gidx(0, g, cl)] = c.tu(i);
        if (b.cmax && g >= 1 && g <= nA + 2) b.cmax[gidx(0, g, cl)] = c.cm(i);
      }
      if (sfrozen[cl] != 0u) continue;
      const bool interior = (i >= 1 && i <= nA);
      double temperature = c.x(F_T, i) / c.tu(i);
      if (b.heating && interior) temperature = tile_heated(b, temperature, dt, gidx(0, g, cl), tile.c0 + cl);
      double l[NS + 1], nd[NS + 1], N = 0.0;
#pragma unroll
      for (int s = 0; s < NS; ++s) l[s] = c.x(F_LNS + s, i);
      l[NS] = c.x(F_LRHO, i);
      exp_n(l, nd);
      bool finite = isfinite(nd[NS]) && isfinite(temperature);
      b.rho[gidx(0, g, cl)] = nd[NS];
      b.temperature[gidx(0, g, cl)] = temperature;
#pragma unroll
      for (int d = 0; d < 3; ++d) b.velocity[gidx(d, g, cl)] = c.x(F_VE + d, i);
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double ws = c.x(F_W + s, i);
        finite = finite && isfinite(nd[s]) && isfinite(ws);
        N = N + nd[s];
        b.vert_vel[gidx(s, g, cl)] = ws;
        b.ndensity_s[gidx(s, g, cl)] = nd[s];
      }
      if (b.log_ns) {
#pragma unroll
        for (int s = 0; s < NS; ++s) b.log_ns[gidx(s, g, cl)] = l[s];
      }
      if (b.ndensity) b.ndensity[gidx(0, g, cl)] = N;
      if (prm.use_ion_advection) {
        const bool pc = in_pcells(i, nA), improved = prm.use_improved_ion_advection != 0;
        double e = 0.0;
#pragma unroll 3
        for (int s = 0; s < NI; ++s) {
          const bool here = s < NADV || pc;
          double v = here ? c.ion(s, i) : b.idensity_s[gidx(s, g, cl)];  // unchanged interior value
          if (here && !improved) v = exp_sl(v);
          const double was = v;
          if (improved && interior && v < 1) v = 1.0;
          finite = finite && isfinite(v);
          if (here || v != was) b.idensity_s[gidx(s, g, cl)] = v;
          e = e + v;
        }
        b.idensity_s[gidx(NI, g, cl)] = e;
      }
      if (!finite) atomicOr(&sst[cl], GITM_ST_NONFINITE);
    }
    __syncthreads();

    if (tid < nc) {
      const int64_t gcol = M.col_offset + tile.c0 + tid;
      uint32_t w = sst[tid];
      if (sfrozen[tid]) w |= GITM_ST_NEG_DENSITY;
      if (dry) w &= GITM_ST_NEG_DENSITY | GITM_ST_NEG_ION_TOP;  // what stops a gather or a boundary pass
      if (w) kp.status[gcol] |= w;
    }
    __syncthreads();
  }
  if (wid == 0) tm_free<512>(tm_base);
}

}  // namespace gv
