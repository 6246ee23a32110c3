// vert_adjoint.cuh -- reverse-mode derivative of one vertical step (Rusanov
// solver, GITM-array form): gitm_vert_plan_adjoint.
//
// The reference has no adjoint; this is the hand-written reverse of the
// forward kernel of vert_kernel.cuh, statement by statement, with every
// branch (limiter case, clamp, boundary switch, max of |w|) differentiated on
// the side the forward took.
//
// One CTA per tile of columns, persistent over tiles.  The states it needs --
// the gathered state, the post-boundary stage inputs X0..X3 and the final X4
// -- come from the saving step (vert_tile.cuh), run by the caller, or ahead of
// this kernel a few thousand columns at a time.  The reverse sweep runs from
// the scatter back to the gather:
//   scatter^T -> bc^T(X4) -> RK combination^T -> for k = 3..0:
//     load X_k, recompute its slopes, stage_k^T at every interior cell
//     (one thread per cell writes its own cell's adjoint; the sweeps'
//     shares of the neighbouring cells go by shuffles within a warp, through
//     a small edge buffer across warps; GradLogConS's are left in shared
//     memory), the gather of those shares (one thread per cell), slopes^T
//     (one thread per field and run of cells), bc^T(X_k) and the
//     combination^T of X_k
//   -> bc^T(X0) -> gather^T and producers^T.
// Shared memory per column: the state, its adjoint, the slopes and their
// adjoints, the per-cell coefficients and their adjoints.  Tensor memory: the
// adjoints of New, of the RK accumulators and of Orig.
//
// What bounds it: chains and the arrival of instructions at 8 warps per SM
// (255 registers a thread); the FP64 pipe is a quarter busy.  A 2.5 degree
// rollout (4 steps, checkpoints every 2, 10,368 columns) 16.3 -> 14.1 ms, one
// step forward and backward of 2,592 columns 1.30 -> 1.14 ms with tensor
// memory for global scratch and Orig's adjoint, the boundary split in three,
// slopes^T by faces, edge shares a thread each and the species' sweep adjoints
// in a loop (220 -> 198 KB of code).
#pragma once

#include "vert_kernel.cuh"
#include "vert_tmem.cuh"

namespace gv {

struct AdjLayout {
  Layout L;  // X0: the state; X1: its adjoint
  int DB, GU, FB, CMB, GMB, TUB, MMB, LC, stride;
};

__host__ __device__ inline AdjLayout make_adj_layout(int nAlts) {
  AdjLayout A;
  A.L = make_layout(nAlts);
  // no Orig region: its adjoint is in tensor memory
  const int cut = A.L.DL - A.L.O;
  A.L.DL -= cut;
  A.L.TU -= cut;
  A.L.CM -= cut;
  A.L.GM -= cut;
  A.L.SC -= cut;
  A.L.stride -= cut;
  const int G = nAlts + 4;
  int o = A.L.stride;
  A.DB = o;  o += NSTENCIL * (nAlts + 2);
  // GradLogConS's -Eddy vb_s of interior cell i at [s * nAlts + i - 1], and
  // their sum (for LogRho) at s = NS: cell_gather hands them to the
  // neighbouring cells
  A.GU = o;  o += (NS + 1) * nAlts;
  // the dissipation coefficients' adjoints of interior cell i (halved): its
  // lower face at [i - 1], its upper face at [nAlts + i - 1]
  A.FB = o;  o += 2 * nAlts;
  A.CMB = o; o += G;
  A.GMB = o; o += G;
  A.TUB = o; o += G;
  A.MMB = o; o += 4;  // MeanMajorMass at cells -1, 0; the heating-factor sum
  A.LC = o;  o += (NSTENCIL * (nAlts + 2) + 7) / 8;  // limiter branch per slope, one byte each
  A.stride = o;
  return A;
}

constexpr int ADJ_NSTATE = 6;    // gathered state, X0, X1, X2, X3, X4
// threads per CTA of the adjoint kernel (2 columns of 50 cells per CTA; 64
// threads with one column measured 3 % slower)
constexpr int ADJ_THREADS = 128;
// The stage adjoint's shares that cross a warp boundary inside a column: per
// boundary (lane 31 of warp b | lane 0 of warp b+1) and swept field, the
// value and slope shares to the right cell and to the left cell.
constexpr int ADJ_EDGE_DOUBLES = (ADJ_THREADS / 32 - 1) * NSTENCIL * 4;

// Tensor memory of a thread, 128 doubles: the adjoints of the stage's New,
// the combination's accumulators and the adjoint of Orig at the thread's cell
// (three blocks of 20 for the 19 fields, read as groups of 8, 8 and 4), then
// the thread's share of Orig's adjoint at the ghost and passive-ion cells and
// four values per species of the stage adjoint.
// Two CTAs fill an SM's.  In global scratch and shared memory they left 28 KB
// of L1, which the scratch itself (78 KB) and the grid's rows (24 KB) shared.
constexpr int ADJ_TM_K = 0, ADJ_TM_ACC = 40, ADJ_TM_O = 80, ADJ_TM_OG = 120, ADJ_TM_SP = 136, ADJ_TM_COLS = 256;
constexpr int ADJ_OG = NF * 4 + NPAS * NPC;  // ghost and passive-ion cells of a column
static_assert(ADJ_TM_OG + 2 * ((ADJ_THREADS / 32 * ADJ_OG + ADJ_THREADS - 1) / ADJ_THREADS) <= ADJ_TM_SP &&
                  ADJ_TM_SP + 8 * NS <= ADJ_TM_COLS,
              "a CTA of at most ADJ_THREADS / 32 columns");

// The columns' slots, the edge shares, then the status words.
__host__ __device__ inline size_t adj_smem_bytes(int nAlts, int nc) {
  return (size_t(make_adj_layout(nAlts).stride) * nc + ADJ_EDGE_DOUBLES) * sizeof(double) +
         size_t(nc) * 2 * sizeof(uint32_t);
}

// Defined in vert_adjoint.cu (the kernel's own translation unit).
const void* adjoint_kernel_fn();
const void* adjoint_kernel_fn_n50();  // members of exactly 50 altitudes
cudaError_t adjoint_set_consts(const Consts& k);
cudaError_t adjoint_set_consts_n50(const Consts& k);
__host__ __device__ inline int adj_state_doubles(int nAlts) { return NF * (nAlts + 4) + NPAS * NPC; }

constexpr int ADJ_INLINE_BARS = 4;  // members whose descriptors travel in the kernel parameters

struct AParams {
  const DevMember* members;
  const GitmColumnAdjoint* bars;      // device array (more members than fit inline)
  GitmColumnAdjoint bars_inline[ADJ_INLINE_BARS];
  int n_inline;                       // > 0: use bars_inline
  const Tile* tiles;
  int n_tiles;
  int per_max;             // adj_state_doubles of the largest member
  double dt;
  uint32_t* status;
  GitmVertParams prm;
  // states saved by the saving step kernel, state s of the plan's column c at
  // saved[(s * saved_ncols + c - saved_c0) * per_max]
  const double* saved;
  int64_t saved_ncols;
  int64_t saved_c0;
};

// ---------------------------------------------------------------- helpers
// The branch of limiter_mc (ModLimiter.f90:16-36) at (u, d) that its
// derivative follows: 0 a zero slope, 1 the slope is beta u, 2 it is beta d,
// 3 it is the mean (u + d) / 2 (ties go to the first candidate of the
// forward's min / max).  The slope's adjoint ob then gives u the adjoint
// beta ob (1) or ob / 2 (3), and d beta ob (2) or ob / 2 (3).
__device__ __forceinline__ int limiter_mc_branch(double u, double d, double beta) {
  const double bu = fabs(beta * u), bd = fabs(beta * d), av = fabs((u + d) * 0.5);
  const bool pos = (u > 0.0) && (d > 0.0);
  const bool neg = !(u > 0.0) && (d < 0.0);
  const bool first = bu <= bd;
  return (pos || neg) ? ((first ? bu : bd) <= av ? (first ? 1 : 2) : 3) : 0;
}

// Where a cell's neighbour is held in the stage adjoint: the next lane of
// the same warp, a ghost cell (no thread; only this cell gives it shares
// there), or a cell of the neighbouring warp.
enum NbKind : int { NB_LANE = 0, NB_GHOST = 1, NB_WARP = 2 };

// Per-column view of the adjoint arrays in shared memory.
struct ColAdj {
  double* xb;    // adjoint of the state, [f*G + cell+1]
  double* xbp;   // its passive-ion cells
  double* db;    // slope adjoints [f*(nAlts+2) + cell]
  double* gu;    // GradLogConS's -Eddy vb_s [s*nAlts + i-1]; their sum at s = NS
  double* fb;    // the dissipation coefficients' adjoints, halved [i-1], [nAlts + i-1]
  double* cmb;   // cMax adjoint [cell+1]
  double* gmb;   // Gamma adjoint
  double* tub;   // TempUnit adjoint
  double* mmb;   // MeanMajorMass(-1), MeanMajorMass(0), heating-factor sum
  uint8_t* lc;   // limiter branch of each slope [f*(nAlts+2) + cell] (limiter_mc_branch)
  int G, nA;
  // the stage adjoint of interior cells (one thread per cell): where this cell's neighbours are, the CTA's edge
  // shares and this thread's warp
  bool act;  // this lane has a cell (the idle lanes of a warp repeat the last one and write nothing)
  int nbl, nbr;
  double* eb;
  int wid;

  __device__ __forceinline__ double& x(int f, int i) const { return xb[f * G + i + 1]; }
  __device__ __forceinline__ double& ion(int s, int i) const {
    return (s < NADV) ? xb[(F_I + s) * G + i + 1] : xbp[(s - NADV) * NPC + pcell(i, nA)];
  }
  // In the stage adjoint the value and slope adjoints of interior cell i
  // are written by its own thread alone (the neighbours' shares reach it by
  // shuffles, or later through cell_gather), those of the ghost cells by
  // the end cells' threads alone.
  __device__ __forceinline__ void own(int f, int i, double v) const {
    if (act) xb[f * G + i + 1] += v;
  }
  // a sweep's value share xv and slope share dv for neighbour cell j of kind
  // nb (not NB_LANE); side 0: j = i+1, side 1: j = i-1
  __device__ __forceinline__ void give(int f, int j, double xv, double dv, int nb, int side) const {
    if (nb == NB_GHOST) {
      own(f, j, xv);
      db[f * (nA + 2) + j] += dv;
    } else {
      double* e = eb + ((wid - side) * NSTENCIL + f) * 4 + 2 * side;
      e[0] += xv;
      e[1] += dv;
    }
  }
};

// ---------------------------------------------------------------- boundaries^T
// Reverse of bc_column (set_vertical_bcs.Earth.f90:8-652) in three parts that
// touch disjoint cells and fields and so run in different warps: the lower
// boundary and the upper one's neutrals, 16 lanes per column with lanes over
// species and ions (two columns a warp), and the upper one's ions, a warp per
// column.  c: the post-boundary state; a: its adjoint, replaced by the adjoint
// of the pre-boundary state (ghost cells the boundary overwrites get 0, ghost
// cells it reads before overwriting get their contribution).  The lower part writes the adjoints of cells
// <= 5, the upper ones of cells >= nAlts-4.  With a warp per half column the
// upper half's chain was 10.7 kcycles and the lower one's 5.7; now the ions'
// is 7.9, mostly its instructions' arrival, and the neutrals' 4.5.
__device__ __forceinline__ double half_seq_sum(double v) {  // lane_seq_sum of the species of 16 lanes
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < NS; ++k) s = s + __shfl_sync(0xffffffffu, v, k, 16);
  return s;
}
static_assert(NI < 16, "the idle lanes of a column");

// The upper boundary's neutrals; s: the lane's species, 15 for a lane without a column.
__device__ inline void bc_adjoint_upper(const ColCtx& c, const ColAdj& a, int s) {
  const int nA = c.L.nAlts;
  const double* sc = c.col + c.L.SC;
  auto X = [&](int f, int i) -> double { return c.x(f, i); };
  // lines 598-604: LogRho of the two top ghosts (both cells' sums first)
  {
    double ms1 = 0.0, ms2 = 0.0;
    if (s < NS) {
      ms1 = c_k.mass[s] * exp(X(F_LNS + s, nA + 1));
      ms2 = c_k.mass[s] * exp(X(F_LNS + s, nA + 2));
    }
    const double r1 = half_seq_sum(ms1);
    const double r2 = half_seq_sum(ms2);
    const double lb1 = a.x(F_LRHO, nA + 1), lb2 = a.x(F_LRHO, nA + 2);
    __syncwarp();
    if (s < NS) {
      a.x(F_LNS + s, nA + 1) += lb1 * ms1 / r1;
      a.x(F_LNS + s, nA + 2) += lb2 * ms2 / r2;
    }
    if (s == 0) {
      a.x(F_LRHO, nA + 1) = 0.0;
      a.x(F_LRHO, nA + 2) = 0.0;
    }
  }
  __syncwarp();
  // lines 420-486: species winds and hydrostatic densities, one per lane
  double tb = 0.0;
  if (s < NS) {
    const double T = X(F_T, nA);
    const double wn = X(F_W + s, nA);
    const double w1b = a.x(F_W + s, nA + 1), w2b = a.x(F_W + s, nA + 2);
    a.x(F_W + s, nA + 1) = 0.0;
    a.x(F_W + s, nA + 2) = 0.0;
    if (photochemical(s) && wn < 0.0) {
      a.x(F_W + s, nA) -= w1b;
      a.x(F_W + s, nA - 1) -= w2b;
    } else {
      a.x(F_W + s, nA) += w1b + w2b;
    }
    const double ish1 = (-0.5 * (sc[SC_EG + 3] + sc[SC_EG + 2])) * c_k.mass[s] / (0.5 * (T + T) * KB);
    const double ish2 = (-0.5 * (sc[SC_EG + 4] + sc[SC_EG + 3])) * c_k.mass[s] / (0.5 * (T + T) * KB);
    const double lb2 = a.x(F_LNS + s, nA + 2);
    a.x(F_LNS + s, nA + 2) = 0.0;
    const double l1b = lb2 + a.x(F_LNS + s, nA + 1);
    a.x(F_LNS + s, nA + 1) = 0.0;
    const double ish2b = -sc[SC_DAF + 5] * lb2;
    a.x(F_LNS + s, nA) += l1b;
    const double ish1b = -sc[SC_DAF + 4] * l1b;
    tb = -(ish1b * ish1 + ish2b * ish2) / T;
  }
  tb = half_seq_sum(tb);
  if (s == 0) {
    // lines 466-469: Temp(nA+1:nA+2) = Temp(nA)
    a.x(F_T, nA) += tb + a.x(F_T, nA + 1) + a.x(F_T, nA + 2);
    a.x(F_T, nA + 1) = 0.0;
    a.x(F_T, nA + 2) = 0.0;
    // lines 455-463: Vel_GD up = |Vel_GD up (nA)|
    const double v = X(F_VU, nA);
    const double sg = (v < 0.0) ? -1.0 : (v > 0.0 ? 1.0 : 0.0);
    a.x(F_VU, nA) += sg * (a.x(F_VU, nA + 1) + a.x(F_VU, nA + 2));
    a.x(F_VU, nA + 1) = 0.0;
    a.x(F_VU, nA + 2) = 0.0;
    // lines 420-430: horizontal winds
    for (int f = F_VE; f <= F_VN; ++f) {
      a.x(f, nA) += a.x(f, nA + 1) + a.x(f, nA + 2);
      a.x(f, nA + 1) = 0.0;
      a.x(f, nA + 2) = 0.0;
    }
  }
  __syncwarp();
}

// The upper boundary's ions; pg1, pg2: the pre-boundary values of the lane's
// ion at nAlts+1 and nAlts+2, which the boundary reads.
__device__ inline void bc_adjoint_ions(const ColCtx& c, const ColAdj& a, double pg1, double pg2, const GitmVertParams& prm,
                                       int lane, uint32_t* st) {
  const int nA = c.L.nAlts;
  const double* sc = c.col + c.L.SC;
  const int s = lane;
  auto XI = [&](int q, int i) -> double { return c.ion(q, i); };
  const double* bu = sc + SC_BCC + 10;  // upper mesh coefficients: nA+1 then nA+2
  auto dAF = [&](int i) { return c.dAF(i); };
  // lines 488-596: ions, one per lane.  With UseImprovedIonAdvection the
  // logs of the extrapolation are taken lane-parallel first, as bc_column
  // takes them: lg[7 s + j] = log(pre-boundary ion s at nAlts+2-j), j =
  // 0..6; the ghost values the forward set (exp of its extrapolations) are
  // read from the post-boundary state, and the log of the first one is its
  // exponent y, as bc_column uses it.
  {
    const bool improved = prm.use_improved_ion_advection != 0;
    double tp = 0.0;
    bool neg = false;
    double* lg = c.col + c.L.DL;  // scratch: the slopes are dead during the boundary adjoint
    static_assert(NI * 9 <= NSTENCIL * (8 + 2), "the ion logs and ghosts fit the slope region at nAlts >= 8");
    if (improved) {
#pragma unroll 1
      for (int i = 1 + lane; i <= nA; i += 32) tp += c.dAF(i) * XI(0, i);
      if (s < NI) {
        neg = (pg1 < 0.0) || (pg2 < 0.0);
        for (int q = nA - 5; q <= nA; ++q) neg = neg || (XI(s, q) < 0.0);
        lg[NI * 7 + s] = pg2;
        lg[NI * 8 + s] = pg1;
      }
      __syncwarp();
#pragma unroll 1
      for (int q = lane; q < NI * 7; q += 32) {
        const int si = q / 7, j = q - si * 7;
        const int cell = nA + 2 - j;
        lg[q] = log((j < 2) ? lg[NI * (7 + j) + si] : XI(si, cell));
      }
    } else {
#pragma unroll 1
      for (int i = 1 + lane; i <= nA; i += 32) tp += c.dAF(i) * exp(XI(0, i));
    }
    for (int off = 16; off > 0; off >>= 1) tp += __shfl_xor_sync(0xffffffffu, tp, off);
    // the forward's test (bc_column): TEC < MinTEC * 1e16
    const bool hold = (tp < prm.min_tec * 1e16) && (sc[SC_PLASMA] != 0.0);
    const bool anyneg = __any_sync(0xffffffffu, neg);
    __syncwarp();
    const double dT = dAF(nA);
    if (anyneg) {
      if (lane == 0) atomicOr(st, GITM_ST_ADJ_BRANCH);
    } else if (!hold && s < NI) {
      const double* C = bu;
      const double* D = bu + 5;
      if (improved) {
        const double* n = lg + s * 7 + 1;  // n[k] = log(ion at nAlts+1-k), k = 0..5
        const double g0 = lg[s * 7];
        const double dnr = C[0] * n[1] + C[1] * n[2] + C[2] * n[3] + C[3] * n[4] + C[4] * n[5];
        const double lim = -(0.001 * n[0] / dT);
        const bool t1 = dnr > lim;
        const double dn = t1 ? lim : dnr;
        const double y = n[1] + dn * dAF(nA + 1);
        const double v1 = XI(s, nA + 1);  // exp(y)
        const double dn2r = D[0] * y + D[1] * n[1] + D[2] * n[2] + D[3] * n[3] + D[4] * n[4];
        const double lim2 = -(0.001 * g0 / dT);
        const bool t2 = dn2r > lim2;
        const double v2 = XI(s, nA + 2);  // exp(y + dn2 dAF(nAlts+2))
        double nb[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const double v2b = a.ion(s, nA + 2);
        a.ion(s, nA + 2) = 0.0;
        const double e2 = v2b * v2;
        double yb = e2;
        const double dn2b = e2 * dAF(nA + 2);
        if (t2) {
          a.ion(s, nA + 2) += (dn2b * (-0.001 / dT)) / pg2;
        } else {
          yb += D[0] * dn2b;
          for (int q = 1; q < 5; ++q) nb[q] += D[q] * dn2b;
        }
        const double e1 = a.ion(s, nA + 1) * v1 + yb;
        a.ion(s, nA + 1) = 0.0;
        nb[1] += e1;
        const double dnb = e1 * dAF(nA + 1);
        if (t1) {
          a.ion(s, nA + 1) += (dnb * (-0.001 / dT)) / pg1;
        } else {
          for (int q = 0; q < 5; ++q) nb[q + 1] += C[q] * dnb;
        }
        for (int j = 1; j < 6; ++j) a.ion(s, nA + 1 - j) += nb[j] / XI(s, nA + 1 - j);
      } else {
        const double dn1r = C[0] * XI(s, nA) + C[1] * XI(s, nA - 1) + C[2] * XI(s, nA - 2) +
                            C[3] * XI(s, nA - 3) + C[4] * XI(s, nA - 4);
        const bool t1 = dn1r > -(0.001 * pg1 / dT);
        const double v1 = XI(s, nA + 1);
        const double dn2r = D[0] * v1 + D[1] * XI(s, nA) + D[2] * XI(s, nA - 1) + D[3] * XI(s, nA - 2) +
                            D[4] * XI(s, nA - 3);
        const bool t2 = dn2r > -(0.001 * pg2 / dT);
        const double v2b = a.ion(s, nA + 2);
        a.ion(s, nA + 2) = 0.0;
        double v1b = a.ion(s, nA + 1) + v2b;
        a.ion(s, nA + 1) = 0.0;
        const double dn2b = v2b * dAF(nA + 2);
        if (t2) {
          a.ion(s, nA + 2) += dn2b * (-0.001 / dT);
        } else {
          v1b += D[0] * dn2b;
          for (int q = 1; q < 5; ++q) a.ion(s, nA + 1 - q) += D[q] * dn2b;
        }
        a.ion(s, nA) += v1b;
        const double dn1b = v1b * dAF(nA + 1);
        if (t1) {
          a.ion(s, nA + 1) += dn1b * (-0.001 / dT);
        } else {
          for (int q = 0; q < 5; ++q) a.ion(s, nA - q) += C[q] * dn1b;
        }
      }
    }
  }
  __syncwarp();
}

// The lower boundary; s: the lane's species or ion, 15 for a lane without a column.
__device__ inline void bc_adjoint_lower(const ColCtx& c, const ColAdj& a, const GitmVertParams& prm, int s) {
  const double* sc = c.col + c.L.SC;
  auto X = [&](int f, int i) -> double { return c.x(f, i); };
  const double* bl = sc + SC_BCC;  // lower mesh coefficients: cell 0 then -1
  const bool msis = prm.use_msis_bcs && sc[SC_HASLBC] != 0.0;
  const double* C0 = bl;
  const double* C1 = bl + 5;
  // this lane's species winds of cells 0 and -1 as the extrapolation of
  // lines 334-344 left them (lines 382-395 may flip them afterwards)
  double w0e = 0.0, wm1e = 0.0;
  if (s < NS) {
    const double d0 = X(F_W + s, 1) * C0[0] + X(F_W + s, 2) * C0[1] + X(F_W + s, 3) * C0[2] +
                      X(F_W + s, 4) * C0[3] + X(F_W + s, 5) * C0[4];
    w0e = X(F_W + s, 1) - sc[SC_DAF + 2] * d0;
    const double d1 = w0e * C1[0] + X(F_W + s, 1) * C1[1] + X(F_W + s, 2) * C1[2] + X(F_W + s, 3) * C1[3] +
                      X(F_W + s, 4) * C1[4];
    wm1e = w0e - sc[SC_DAF + 1] * d1;
    // lines 382-395: photochemical sign flip
    if (photochemical(s) && X(F_W + s, 1) > 0.0) {
      a.x(F_W + s, 1) -= a.x(F_W + s, 0) + a.x(F_W + s, -1);
      a.x(F_W + s, 0) = 0.0;
      a.x(F_W + s, -1) = 0.0;
    }
  }
  // lines 364-376: MSIS winds of cell -1
  if (msis && s == 0) {
    for (int f = F_VE; f <= F_VN; ++f) {
      const double b = a.x(f, -1);
      a.x(f, -1) = 0.0;
      a.x(f, 0) += b;
      for (int q = 0; q < 5; ++q) a.x(f, q) += -sc[SC_DAF + 1] * C1[q] * b;
    }
  }
  __syncwarp();
  // lines 348-362: LogRho and bulk vertical wind of cells 0 and -1 (both
  // cells' sums first)
  {
    double ms0 = 0.0, msm = 0.0;
    if (s < NS) {
      ms0 = c_k.mass[s] * exp(X(F_LNS + s, 0));
      msm = c_k.mass[s] * exp(X(F_LNS + s, -1));
    }
    const double r0 = half_seq_sum(ms0);
    const double mw0 = half_seq_sum(ms0 * w0e);
    const double rm = half_seq_sum(msm);
    const double mwm = half_seq_sum(msm * wm1e);
    const double lrb0 = a.x(F_LRHO, 0), vub0 = a.x(F_VU, 0);
    const double lrbm = a.x(F_LRHO, -1), vubm = a.x(F_VU, -1);
    __syncwarp();
    const double rb0 = lrb0 / r0 - vub0 * mw0 / (r0 * r0);
    const double mwb0 = vub0 / r0;
    const double rbm = lrbm / rm - vubm * mwm / (rm * rm);
    const double mwbm = vubm / rm;
    if (s < NS) {
      a.x(F_W + s, 0) += mwb0 * ms0;
      a.x(F_LNS + s, 0) += (rb0 + mwb0 * w0e) * ms0;
      a.x(F_W + s, -1) += mwbm * msm;
      a.x(F_LNS + s, -1) += (rbm + mwbm * wm1e) * msm;
    }
    if (s == 0) {
      a.x(F_LRHO, 0) = 0.0;
      a.x(F_VU, 0) = 0.0;
      a.x(F_LRHO, -1) = 0.0;
      a.x(F_VU, -1) = 0.0;
    }
    __syncwarp();
  }
  // lines 304-310: ions float
  if (s < NI) {
    a.ion(s, 1) += a.ion(s, 0) + a.ion(s, -1);
    a.ion(s, 0) = 0.0;
    a.ion(s, -1) = 0.0;
  }
  // lines 205-272 and 334-344, one species per lane
  double l0b = 0.0, tb = 0.0, mb = 0.0;
  if (s < NS) {
    {  // winds: cell -1 from cell 0 (new), then cell 0 from the interior
      const double b = a.x(F_W + s, -1);
      a.x(F_W + s, -1) = 0.0;
      a.x(F_W + s, 0) += b * (1.0 - sc[SC_DAF + 1] * C1[0]);
      for (int q = 1; q < 5; ++q) a.x(F_W + s, q) += -sc[SC_DAF + 1] * C1[q] * b;
      const double b0 = a.x(F_W + s, 0);
      a.x(F_W + s, 0) = 0.0;
      a.x(F_W + s, 1) += b0 * (1.0 - sc[SC_DAF + 2] * C0[0]);
      for (int q = 1; q < 5; ++q) a.x(F_W + s, 1 + q) += -sc[SC_DAF + 2] * C0[q] * b0;
    }
    if (!photochemical(s)) {
      const double b = a.x(F_LNS + s, -1);
      a.x(F_LNS + s, -1) = 0.0;
      if (s == 0) {
        a.x(F_LNS + s, 0) += b;
      } else {
        l0b = b;
        const double ishb = b * sc[SC_DAF + 0];
        const double mg = -0.5 * (sc[SC_EG + 0] + sc[SC_EG + 1]);
        const double mt = 0.5 * (X(F_T, 0) + X(F_T, -1));
        const double mm = 0.5 * (sc[SC_MMM_0] + sc[SC_MMM_M1]);
        const double ish = mg * mm / (mt * KB);
        mb = ishb * mg / (mt * KB);
        tb = 0.5 * (-ishb * ish / mt);
      }
    } else {
#pragma unroll 1
      for (int k = 1; k >= 0; --k) {
        const int i = -k;
        const double* C = bl + 5 * k;
        const double d = X(F_LNS + s, i + 1) * C[0] + X(F_LNS + s, i + 2) * C[1] + X(F_LNS + s, i + 3) * C[2] +
                         X(F_LNS + s, i + 4) * C[3] + X(F_LNS + s, i + 5) * C[4];
        const double up = X(F_LNS + s, i + 1);
        const double dF = sc[SC_DAF + 2 + i];
        double v = up - dF * d;
        const bool flat = d <= 0.0;
        if (flat) v = up;
        const bool floor = (s == 4) && (v < up - 0.333);
        const double b = a.x(F_LNS + s, i);
        a.x(F_LNS + s, i) = 0.0;
        a.x(F_LNS + s, i + 1) += b;
        if (!flat && !floor) {
          const double dbv = -dF * b;
          for (int q = 0; q < 5; ++q) a.x(F_LNS + s, i + 1 + q) += C[q] * dbv;
        }
      }
    }
  }
  mb = half_seq_sum(mb);
  tb = half_seq_sum(tb);
  if (s == 0) {
    a.mmb[0] += 0.5 * mb;
    a.mmb[1] += 0.5 * mb;
    a.x(F_T, 0) += tb;
    a.x(F_T, -1) += tb;
    // lines 192-196
    for (int f : {F_T, F_VE, F_VN, F_VU}) {
      a.x(f, 0) += a.x(f, -1);
      a.x(f, -1) = 0.0;
    }
    // lines 112-148
    a.x(F_VU, 0) = 0.0;
    a.x(F_VE, 0) = 0.0;
    a.x(F_VN, 0) = 0.0;
    if (msis) {
      a.x(F_T, 0) = 0.0;
      a.x(F_LRHO, 0) = 0.0;
      a.x(F_LRHO, -1) = 0.0;
    }
  }
  if (s < NS) {
    a.x(F_W + s, 0) = 0.0;
    a.x(F_W + s, -1) = 0.0;
    if (msis) {
      a.x(F_LNS + s, -1) = 0.0;
      a.x(F_LNS + s, 0) = l0b;
    } else {
      a.x(F_LNS + s, 0) += l0b;
    }
  }
  __syncwarp();
}

// ---------------------------------------------------------------- stage^T
// Reverse of rusanov_cell at interior cell i, in two passes that each hold
// only their own part of the cell's values (one pass over everything held
// the friction matrix, the species terms and all field adjoints at once and
// spilled): cell_adjoint_species (continuity and momentum of the species,
// the friction solve, LogRho) and cell_adjoint_rest (temperature, the
// horizontal winds, the bulk vertical wind's own terms, the ions).  kb:
// the tensor memory of the adjoints of New (the caller applies K = New - state);
// contributions go to the state adjoint (this cell and its neighbours), the
// slope adjoints, the cMax and Gamma adjoints.  Every sweep adjoint is
// linear in its inputs, so the two passes' shares of the temperature
// sweep add up.

// The face geometry of cell i and its sweep (calc_rusanov_alts_rusanov,
// vertical_solver_rusanov.f90:694-718), forward and reverse.
struct CellFaces {
  double dF0, dF1, idc, fc0, fc1;
  double hF0, hF1, hidc;  // the halves of dF0, dF1, idc (a product with 0.5 is exact)
  double fc0b, fc1b;  // adjoints of the two dissipation coefficients

  __device__ __forceinline__ CellFaces(const ColCtx& c, int i) {
    dF0 = c.dAF(i);
    dF1 = c.dAF(i + 1);
    idc = c.g(GC_IDC, i);
    hF0 = 0.5 * dF0;
    hF1 = 0.5 * dF1;
    hidc = 0.5 * idc;
    fc0 = 0.5 * fmax(c.cm(i - 1), c.cm(i));
    fc1 = 0.5 * fmax(c.cm(i), c.cm(i + 1));
    fc0b = 0.0;
    fc1b = 0.0;
  }
  __device__ __forceinline__ void sweep(const ColCtx& c, int f, int i, double& grad, double& diff) const {
    const double* v = &c.col[c.xo + f * c.L.G + 1];
    const double* d = &c.col[c.L.DL + f * (c.L.nAlts + 2)];
    const double L0 = fma(d[i - 1], hF0, v[i - 1]);
    const double R0 = fma(-d[i], hF0, v[i]);
    const double L1 = fma(d[i], hF1, v[i]);
    const double R1 = fma(-d[i + 1], hF1, v[i + 1]);
    grad = (L1 + R1 - L0 - R0) * hidc;
    diff = (fc1 * (R1 - L1) - fc0 * (R0 - L0)) * idc;
  }
  // (gb, dbv) -> faces -> values and slopes; returns this cell's value
  // share, with what the neighbouring cells of the same warp give it (by
  // shuffles), and adds its slope share with theirs; the shares of ghost
  // cells and of cells in the neighbouring warp go by give().
  __device__ __forceinline__ double sweep_adj(const ColCtx& c, const ColAdj& a, int f, int i, double gb,
                                              double dbv) {
    const double* v = &c.col[c.xo + f * c.L.G + 1];
    const double* d = &c.col[c.L.DL + f * (c.L.nAlts + 2)];
    const double L0 = fma(d[i - 1], hF0, v[i - 1]);
    const double R0 = fma(-d[i], hF0, v[i]);
    const double L1 = fma(d[i], hF1, v[i]);
    const double R1 = fma(-d[i + 1], hF1, v[i + 1]);
    const double hg = hidc * gb;
    const double L1b = hg - fc1 * idc * dbv, R1b = hg + fc1 * idc * dbv;
    const double L0b = -hg + fc0 * idc * dbv, R0b = -hg - fc0 * idc * dbv;
    fc1b += idc * (R1 - L1) * dbv;
    fc0b += -idc * (R0 - L0) * dbv;
    const double dl = hF0 * L0b;               // to the slope of cell i-1
    const double dm = -hF0 * R0b + hF1 * L1b;  // this cell's slope
    const double dr = -hF1 * R1b;              // the slope of cell i+1
    const double xr = __shfl_down_sync(0xffffffffu, L0b, 1);  // cell i+1's share of this cell
    const double drr = __shfl_down_sync(0xffffffffu, dl, 1);
    const double xl = __shfl_up_sync(0xffffffffu, R1b, 1);    // cell i-1's
    const double dll = __shfl_up_sync(0xffffffffu, dr, 1);
    double own = R0b + L1b, down = dm;
    if (a.nbl == NB_LANE) {
      own += xl;
      down += dll;
    } else {
      a.give(f, i - 1, L0b, dl, a.nbl, 1);
    }
    if (a.nbr == NB_LANE) {
      own += xr;
      down += drr;
    } else {
      a.give(f, i + 1, R1b, dr, a.nbr, 0);
    }
    if (a.act) a.db[f * (a.nA + 2) + i] += down;
    return own;
  }
  // the dissipation coefficients' adjoints (fc = 0.5 max(cMax, cMax') at
  // each face), kept for cell_gather, which hands them to the cMax of the
  // side each max took; acc: add to what the cell's other pass kept
  __device__ __forceinline__ void keep_fc(const ColAdj& a, int i, bool acc) const {
    if (!a.act) return;
    double& b0 = a.fb[i - 1];
    double& b1 = a.fb[a.nA + i - 1];
    b0 = acc ? b0 + 0.5 * fc0b : 0.5 * fc0b;
    b1 = acc ? b1 + 0.5 * fc1b : 0.5 * fc1b;
  }
};

// Species continuity and momentum (:548-617), the friction solve
// (calc_neutral_friction.f90:47-106), the clamp and LogRho / the bulk wind's
// species terms (:643-658) in reverse.  kb: their New adjoints' tensor memory.  Returns
// the KappaEddyDiffusion adjoint of the cell.
__device__ inline double cell_adjoint_species(const ColCtx& c, const ColAdj& a, int i, const GitmVertParams& prm,
                                              double dt, double eddy, uint32_t kb) {
  CellFaces fa(c, i);
  // ---- forward recompute
  const double invr = c.g(GC_INVR, i), rr = c.g(GC_R, i), grav = c.g(GC_GRAV, i);
  const double T = c.x(F_T, i), VE = c.x(F_VE, i), VN = c.x(F_VN, i);
  const double LR = c.x(F_LRHO, i);
  double gT, dT;
  fa.sweep(c, F_T, i, gT, dT);
  const double itau = 1.0 / (prm.use_damping ? 15 - (1 - exp(-1.0 * c.g(GC_ALT, i) / 1000.0 / 40.0)) * 5.0
                                             : prm.vert_tau);
  const double hz = (VN * VN + VE * VE) * invr;
  const double cor = prm.use_coriolis ? dt * (c.sc(SC_CENT) * rr + c.sc(SC_CORI) * VE) : 0.0;
  double wv[NS], menl[NS];
  double sumrho = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    double gL, dL, gW, dW;
    fa.sweep(c, F_LNS + s, i, gL, dL);
    fa.sweep(c, F_W + s, i, gW, dW);
    const double Ls = c.x(F_LNS + s, i), Ws = c.x(F_W + s, i);
    const double divw = gW + 2 * Ws * invr;
    const double nl = Ls - dt * (divw + Ws * gL) + dt * dL;
    menl[s] = nl;
    const double km = c_k.k_over_m[s];
    double w = Ws - dt * (Ws * gW - hz + T * gL * km + gT * km - grav) + dt * dW - Ws * itau;
    w = w + cor;
    w = w - dt * (prm.thermal_diff_coef[s] * km) * gT;
    wv[s] = w;
  }
  double ns[NS], ir;
  {
    double e[NS];
    exp_n(menl, e);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      menl[s] = c_k.mass[s] * e[s];
      sumrho = sumrho + menl[s];
    }
    double l7[NS + 1], e7[NS + 1];
#pragma unroll
    for (int s = 0; s < NS; ++s) l7[s] = c.x(F_LNS + s, i);
    l7[NS] = -LR;
    exp_n(l7, e7);
#pragma unroll
    for (int s = 0; s < NS; ++s) ns[s] = e7[s];
    ir = e7[NS];
  }
  // reverse of New LogRho = log(sumrho): the continuity adjoints, with
  // New LogNS's own adjoint
  double nlb[NS];
  {
    double k0[8], k2[4];  // LNS and W(1:2); the ions and LogRho
    __syncwarp();
    tm_get(kb, k0);
    tm_get(kb + 2 * F_I, k2);
    const double srb = k2[F_LRHO - F_I] / sumrho;
#pragma unroll
    for (int s = 0; s < NS; ++s) nlb[s] = srb * menl[s] + k0[F_LNS + s];
  }
  double Tb = 0.0, VEb = 0.0, VNb = 0.0, LRb = 0.0, irb = 0.0;
  double nsb[NS], wb[NS], lself[NS];  // lself: GradLogConS's share of this cell's LogNS adjoint
  double eddyb = 0.0;
  // New VU = sum_s w_s m_s ns_s / Rho; New VertVel = the clamped w
  double k0[8] = {}, k1[8] = {};  // W(1:2); W(3:6) and VU
  auto kw = [&](int s) { return s < 2 ? k0[F_W + s] : k1[F_W + s - 8]; };
  if (prm.use_neutral_friction) {
    // the friction solve (friction_solve): S v = M n w
    double glc[NS], mn[NS], vsol[NS], pe[NS];
    grad_log_cons(c, i, glc);
    {
      const double lt = log_sl(T);
      double le[NS];
#pragma unroll
      for (int e = 0; e < NS; ++e) le[e] = c_k.one_minus_e[e] * lt;
      exp_n(le, pe);
    }
#pragma unroll
    for (int e = 0; e < NS; ++e) pe[e] = (dt * c_k.kpair[e]) * pe[e];
#pragma unroll
    for (int s = 0; s < NS; ++s) mn[s] = c_k.mass[s] * ns[s];
    const double shift = friction_range(ns, mn, pe);
#pragma unroll
    for (int s = 0; s < NS; ++s) vsol[s] = mn[s] * wv[s];
    FrictionLdl ldl;
    ldl.factor(ns, mn, pe);
    ldl.eliminate(vsol);
    ldl.back(vsol);
    auto densities = [&] {  // the cell's own again
#pragma unroll
      for (int s = 0; s < NS; ++s) ns[s] = exp_any(c.x(F_LNS + s, i));
    };
    if (shift != 0.0) densities();
    // clamp, bulk wind and their reverse
    __syncwarp();
    tm_get(kb, k0);
    tm_get(kb + 16, k1);
    const double kvu = k1[F_VU - 8];
    double vb[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double v = vsol[s] + (-eddy * glc[s]);
      const bool inside = !(v < -prm.max_vertical_velocity) && !(v > prm.max_vertical_velocity);
      double wc = (v > -prm.max_vertical_velocity) ? v : -prm.max_vertical_velocity;
      wc = (wc < prm.max_vertical_velocity) ? wc : prm.max_vertical_velocity;
      const double m = c_k.mass[s];
      const double wcb = kvu * (m * ns[s] * ir) + kw(s);
      nsb[s] = kvu * wc * m * ir;
      irb += kvu * wc * m * ns[s];
      vb[s] = inside ? wcb : 0.0;
      eddyb -= vb[s] * glc[s];
    }
    // GradLogConS: 5-point mesh on log(m_s) + LogNS - LogRho.  This
    // cell's own share here; u_s = -Eddy vb_s (and their sum, for LogRho)
    // left for cell_gather, which gives cells i-2, i-1, i+1, i+2 theirs
    {
      const double mc = c.g(GC_M0 + 2, i);
      double lrb = 0.0, ul = 0.0;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double u = -eddy * vb[s];
        if (a.act) a.gu[s * a.nA + i - 1] = u;
        ul += u;
        const double v = u * mc;
        lrb -= v;
        lself[s] = v;
      }
      if (a.act) a.gu[NS * a.nA + i - 1] = ul;
      LRb += lrb;
    }
    // (I + dt C) = (M n)^-1 S, so its transpose's solve is wb = M n y with S y = vb
#pragma unroll
    for (int s = 0; s < NS; ++s) wb[s] = vb[s];
    ldl.forward(wb);
    ldl.back(wb);
    if (shift != 0.0) {
      // a density times y is the same at either scale
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        pe[s] *= shift;
        ns[s] = mn[s] * c_k.inv_mass[s];
      }
    }
    // each pair (r, q) through its coefficient P = dt kpair T^(1-e), with y:
    // n_q takes P n_r y_r (v_q - v_r), n_r takes P n_q y_q (v_r - v_q), and log T
    // (1 - e) n_r n_q of both
    double ltb = 0.0;
#pragma unroll
    for (int r = 1; r < NS; ++r)
#pragma unroll
      for (int q = 0; q < r; ++q) {
        const double P = pe[exp_index(r, q)];
        const double t = P * (vsol[q] - vsol[r]);
        const double ar = wb[r] * t, aq = -wb[q] * t;
        nsb[q] = fma(ns[r], ar, nsb[q]);
        nsb[r] = fma(ns[q], aq, nsb[r]);
        ltb = fma(c_k.one_minus_e[exp_index(r, q)] * (ns[r] * ns[q]), ar + aq, ltb);
      }
#pragma unroll
    for (int s = 0; s < NS; ++s) wb[s] *= mn[s];
    Tb += (shift != 0.0 ? ltb / shift : ltb) / T;
    if (shift != 0.0) densities();
  } else {
    __syncwarp();
    tm_get(kb, k0);
    tm_get(kb + 16, k1);
    const double kvu = k1[F_VU - 8];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double v = wv[s];
      const bool inside = !(v < -prm.max_vertical_velocity) && !(v > prm.max_vertical_velocity);
      double wc = (v > -prm.max_vertical_velocity) ? v : -prm.max_vertical_velocity;
      wc = (wc < prm.max_vertical_velocity) ? wc : prm.max_vertical_velocity;
      const double m = c_k.mass[s];
      const double wcb = kvu * (m * ns[s] * ir) + kw(s);
      nsb[s] = kvu * wc * m * ir;
      irb += kvu * wc * m * ns[s];
      wb[s] = inside ? wcb : 0.0;
      lself[s] = 0.0;
      if (a.act) a.gu[s * a.nA + i - 1] = 0.0;
    }
    if (a.act) a.gu[NS * a.nA + i - 1] = 0.0;
  }
  // species momentum, continuity and their sweeps
  double gTb = 0.0, hzb = 0.0, corb = 0.0;
  // (a loop, its inputs by way of tensor memory: unrolled over the species it
  // was 6 times the code, and the stage waits for its instructions)
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double v[4] = {wb[s], nlb[s], fma(nsb[s], ns[s], lself[s]), 0.0};
    tm_put(kb + (ADJ_TM_SP - ADJ_TM_K) + 8 * s, v);
  }
  tm_put_wait();
#pragma unroll 1
  for (int s = 0; s < NS; ++s) {
    double in[4];
    __syncwarp();
    tm_get(kb + (ADJ_TM_SP - ADJ_TM_K) + 8 * s, in);
    double gL, dL, gW, dW;
    fa.sweep(c, F_LNS + s, i, gL, dL);
    fa.sweep(c, F_W + s, i, gW, dW);
    const double Ws = c.x(F_W + s, i);
    const double km = c_k.k_over_m[s];
    const double w = in[0];
    double Wb = w * (1.0 - dt * gW - itau);
    double gWb = -dt * Ws * w;
    hzb += dt * w;
    Tb += -dt * gL * km * w;
    double gLb = -dt * T * km * w;
    gTb += -dt * km * w - dt * (prm.thermal_diff_coef[s] * km) * w;
    const double dWb = dt * w;
    corb += w;
    // New LogNS = nl = Ls - dt (divw + Ws gL) + dt dL
    const double n = in[1];
    double Lb = in[2] + n;
    const double divwb = -dt * n;
    Wb += -dt * gL * n + 2 * invr * divwb;
    gLb += -dt * Ws * n;
    const double dLb = dt * n;
    gWb += divwb;
    Lb += fa.sweep_adj(c, a, F_LNS + s, i, gLb, dLb);
    Wb += fa.sweep_adj(c, a, F_W + s, i, gWb, dWb);
    a.own(F_LNS + s, i, Lb);
    a.own(F_W + s, i, Wb);
  }
  LRb -= irb * ir;
  if (prm.use_coriolis) VEb += corb * dt * c.sc(SC_CORI);
  VNb += hzb * 2 * VN * invr;
  VEb += hzb * 2 * VE * invr;
  // the species' share of the temperature sweep
  Tb += fa.sweep_adj(c, a, F_T, i, gTb, 0.0);
  fa.keep_fc(a, i, false);
  a.own(F_T, i, Tb);
  a.own(F_VE, i, VEb);
  a.own(F_VN, i, VNb);
  a.own(F_LRHO, i, LRb);
  return eddyb;
}

// Temperature, horizontal winds, the bulk vertical wind's own terms and the
// ions (:557-568, :660-680) in reverse.
__device__ inline void cell_adjoint_rest(const ColCtx& c, const ColAdj& a, int i, double dt, double ivup,
                                         uint32_t kb) {
  // the New adjoints this pass reads
  double k1[8], ki[4];
  tm_get(kb + 16, k1);
  tm_get(kb + 2 * F_I, ki);
  const double kE = k1[F_VE - 8], kN = k1[F_VN - 8], kT = k1[F_T - 8];
  CellFaces fa(c, i);
  const double invr = c.g(GC_INVR, i);
  const double T = c.x(F_T, i), VU = c.x(F_VU, i);
  const double gm = c.gm(i);
  double gT, dT, gE, dE, gN, dN, gU, dU;
  fa.sweep(c, F_T, i, gT, dT);
  fa.sweep(c, F_VE, i, gE, dE);
  fa.sweep(c, F_VN, i, gN, dN);
  fa.sweep(c, F_VU, i, gU, dU);
  const double divv = gU + 2 * VU * invr;
  // ions: New = I - dt (IVel gI) + dt dI
#pragma unroll
  for (int s = 0; s < NADV; ++s) {
    const double k = ki[s];
    const double own = fa.sweep_adj(c, a, F_I + s, i, -dt * ivup * k, dt * k);
    a.own(F_I + s, i, k + own);
  }
  // horizontal winds: New = V - dt VU gV + dt dV
  double VEb = kE + fa.sweep_adj(c, a, F_VE, i, -dt * VU * kE, dt * kE);
  double VNb = kN + fa.sweep_adj(c, a, F_VN, i, -dt * VU * kN, dt * kN);
  double VUb = -dt * gE * kE - dt * gN * kN;
  // temperature: New = T - dt (VU gT + (Gamma - 1) T divv) + dt dT
  double Tb = kT;
  VUb += -dt * gT * kT;
  const double gTb = -dt * VU * kT;
  const double gmb = -dt * T * divv * kT;
  Tb += -dt * (gm - 1.0) * divv * kT;
  const double divvb = -dt * (gm - 1.0) * T * kT;
  VUb += 2 * invr * divvb;
  Tb += fa.sweep_adj(c, a, F_T, i, gTb, dt * kT);
  VUb += fa.sweep_adj(c, a, F_VU, i, divvb, 0.0);
  fa.keep_fc(a, i, true);
  if (a.act) a.gmb[i + 1] += gmb;
  a.own(F_T, i, Tb);
  a.own(F_VE, i, VEb);
  a.own(F_VN, i, VNb);
  a.own(F_VU, i, VUb);
}

// The limited slopes of cell i (interior: 4th-order form; cells 0 and
// nAlts+1: 2nd-order form), as rusanov_slopes_cell forms them, with each
// slope's limiter branch recorded for slopes_adjoint_run.
__device__ inline void slopes_with_branches(const ColCtx& c, const ColAdj& a, int i, double beta) {
  const int nA = c.L.nAlts;
  const bool end = (i == 0 || i == nA + 1);
  const double cu = end ? c.g(GC_IDF, i + 1) : c.g(GC_H2, i + 1);
  const double cd = end ? c.g(GC_IDF, i) : c.g(GC_H2, i);
  // both forms in one expression, as rusanov_slopes_cell
  const double fa = end ? 1.0 : F1, fb = end ? 0.0 : F2;
  const int ip2 = min(i + 2, nA + 2), im2 = max(i - 2, -1);
  // state, slopes and branch bytes are disjoint regions (restrict: the
  // loads of later fields may be issued ahead of earlier stores)
  const double* __restrict__ xv = c.col + c.xo + 1;
  double* __restrict__ sl = c.col + c.L.DL + i;
  uint8_t* __restrict__ br = a.lc + i;
#pragma unroll 3
  for (int f = 0; f < NSTENCIL; ++f) {
    const double* v = xv + f * c.L.G;
    const double u = cu * (fa * (v[i + 1] - v[i]) - fb * (v[ip2] - v[i - 1]));
    const double d = cd * (fa * (v[i] - v[i - 1]) - fb * (v[i + 1] - v[im2]));
    sl[f * (nA + 2)] = limiter_mc(u, d, beta);
    br[f * (nA + 2)] = uint8_t(limiter_mc_branch(u, d, beta));
  }
}

// Adjoint of the limited slopes into the state adjoint, on the branches
// slopes_with_branches recorded.  With E_i = F1 (v[i+1] - v[i]) - F2 (v[i+2] - v[i-1])
// at the face between cells i and i+1, the slope of interior cell i is the
// limiter of u = H2(i+1) E_i and d = H2(i) E_(i-1), so the face's adjoint is
// H2(i+1) (ub(i) + db(i+1)): what slope i gives its upper difference and slope
// i+1 its lower one, each by its branch.  The 2nd-order differences of cells 0
// and nAlts+1 are the faces' s.  Cell j then takes the faces j-2 .. j+1.  One
// thread walks the faces of field f and owns the state cells j0..j1 (within
// -1..nAlts+2); a cell is written once (no atomics).  10.2 kcycles per stage
// with the five shares of every slope, 6.8 by faces, four at a time with their
// loads ahead of the stores.
__device__ inline void slopes_adjoint_run(const ColCtx& c, const ColAdj& a, int f, int j0, int j1, double beta) {
  const int nA = c.L.nAlts;
  const double* __restrict__ dbp = a.db + f * (nA + 2);
  const uint8_t* __restrict__ lcp = a.lc + f * (nA + 2);
  // the state adjoint of field f (a region apart from the inputs: the loads
  // of later cells may go ahead of the stores)
  double* __restrict__ xo = a.xb + f * a.G + 1;
  double ub = 0.0;  // slope i's share of its upper difference
  {
    const int i = j0 - 2;
    if (i >= 1) {  // j0 - 2 <= nAlts
      const int br = lcp[i];
      ub = (br == 1) ? beta * dbp[i] : (br == 3) ? 0.5 * dbp[i] : 0.0;
    }
  }
  double e1 = 0.0, e2 = 0.0, e3 = 0.0;  // the 4th-order adjoints of faces i-1, i-2, i-3
#pragma unroll 1
  for (int i0 = j0 - 2; i0 <= j1 + 1; i0 += 4) {
    double ob[4], h[4], x[4];
    int br[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k, n = min(max(i + 1, 0), nA + 1);
      br[k] = lcp[n];
      ob[k] = dbp[n];
      h[k] = c.g(GC_H2, n);
      x[k] = xo[min(max(i - 1, j0), j1)];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k;
      const double mean = 0.5 * ob[k], one = beta * ob[k];
      const double u = (br[k] == 1) ? one : (br[k] == 3) ? mean : 0.0;
      const double d = (br[k] == 2) ? one : (br[k] == 3) ? mean : 0.0;
      // slopes of interior cells only
      const bool in = i + 1 >= 1 && i + 1 <= nA;
      const double e = h[k] * (ub + (in ? d : 0.0));
      ub = in ? u : 0.0;
      if (i - 1 >= j0 && i - 1 <= j1) xo[i - 1] = x[k] + fma(F1, e2 - e1, F2 * (e - e3));
      e3 = e2;
      e2 = e1;
      e1 = e;
    }
  }
  // the 2nd-order differences of cells 0 and nAlts+1: between cells i and i+1
  auto s = [&](int i) -> double {
    const int lo = i + 1, up = i;  // the slope whose lower, upper difference it is
    const int n = (lo == 0 || lo == nA + 1) ? lo : (up == 0 || up == nA + 1) ? up : -1;
    if (n < 0) return 0.0;
    const int br = lcp[n];
    const double ob = dbp[n];
    return c.g(GC_IDF, i + 1) * ((br == 3) ? 0.5 * ob : (br == (n == lo ? 2 : 1)) ? beta * ob : 0.0);
  };
#pragma unroll 1
  for (int k = 0; k < 6; ++k) {
    const int j = k < 3 ? k - 1 : nA + k - 3;
    if (j >= j0 && j <= j1) xo[j] += s(j - 1) - s(j);
  }
}

// The thread whose cell takes side `side` of warp boundary bnd's edge shares
// (0: the right cell, what lane 31 gave it; 1: the left cell, what lane 0 of
// the next warp gave it), -1 where the two cells are of different columns.
__device__ __forceinline__ int edge_thread(int bnd, int side, int nA, int nitems) {
  const int right = 32 * (bnd + 1);
  return (right < nitems && right % nA != 0) ? right - side : -1;
}

// What reaches state cell m (-1..nAlts+2) of one column from the other
// cells after the stage adjoint: GradLogConS's shares (u_s mc_q of interior
// cell j = m - q + 2, q != 2, to LogNS_s; -sum_s u_s mc_q to LogRho),
// cMax's, and, when cell m and its neighbour sit on the two sides of a warp
// boundary, the LogNS sweeps' value shares of the edge buffer (the other
// fields' and the slopes' are added by a thread each, next to this).
// t0: the thread of the column's cell 1; nitems: threads holding cells.
__device__ inline void cell_gather(const ColCtx& c, const ColAdj& a, int m, int t0, int nitems) {
  const int nA = c.L.nAlts;
  int edge = -1;  // 2 boundary + side
  {
    const int t = t0 + m - 1, lane = t & 31;
    const int bnd = (t >> 5) - (lane == 0 ? 1 : 0), side = lane == 0 ? 0 : 1;
    if (m >= 1 && m <= nA && (lane == 0 || lane == 31) && bnd >= 0 && edge_thread(bnd, side, nA, nitems) == t)
      edge = 2 * bnd + side;
  }
  double mc[4];
  int jj[4];
  bool ok[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int d = (k < 2) ? k - 2 : k - 1;  // source cell m + d, d = -2, -1, 1, 2
    const int j = m + d;
    ok[k] = (j >= 1 && j <= nA);
    jj[k] = ok[k] ? j : 1;
    mc[k] = ok[k] ? c.g(GC_M0 + 2 - d, j) : 0.0;
  }
#pragma unroll
  for (int s = 0; s <= NS; ++s) {
    const double* u = a.gu + s * nA - 1;
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) v += ok[k] ? u[jj[k]] * mc[k] : 0.0;
    if (s < NS && edge >= 0) v += a.eb[(edge >> 1) * (NSTENCIL * 4) + (F_LNS + s) * 4 + 2 * (edge & 1)];
    a.x((s < NS) ? F_LNS + s : F_LRHO, m) += (s < NS) ? v : -v;
  }
  // cMax of cell m: the dissipation coefficients of the faces whose max
  // took it (cells m and m+1 at their lower faces, cells m-1 and m at their
  // upper faces), in that order
  {
    double cb = 0.0;
    const double cmm = c.cm(m - (m > -1 ? 1 : 0)), cm0 = c.cm(m), cmp = c.cm(m + (m < nA + 2 ? 1 : 0));
    if (m + 1 >= 1 && m + 1 <= nA && cm0 >= cmp) cb += a.fb[m];              // cell m+1, lower face
    if (m >= 1 && m <= nA && !(cmm >= cm0)) cb += a.fb[m - 1];               // cell m, lower face
    if (m >= 1 && m <= nA && cm0 >= cmp) cb += a.fb[nA + m - 1];             // cell m, upper face
    if (m - 1 >= 1 && m - 1 <= nA && !(cmm >= cm0)) cb += a.fb[nA + m - 2];  // cell m-1, upper face
    a.cmb[m + 1] += cb;
  }
}

// 8-byte asynchronous global -> shared copy (cp.async: no register round
// trip, every copy of a thread in flight at once); cp_async_wait_all waits
// for the calling thread's copies.
__device__ __forceinline__ void cp_async8(double* smem_dst, const double* gsrc) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---------------------------------------------------------------- the kernel
// NA > 0: every member has exactly NA altitudes (the host checks), so the
// layout offsets and loop bounds are compile-time constants; NA = 0 reads
// nAlts from the member.
static_assert((ADJ_THREADS / 32 - 1) * NSTENCIL * 2 <= ADJ_THREADS && F_LNS == 0, "a thread per edge share");

template <int NT, int NA = 0>
__global__ void __launch_bounds__(NT, 1) vert_adjoint_kernel(const AParams kp) {
  static_assert(NT == ADJ_THREADS, "the edge-share buffer is sized for ADJ_THREADS");
  extern __shared__ double sm[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int wid = tid >> 5;
  constexpr int nw = NT / 32;
  const GitmVertParams& prm = kp.prm;
  const double dt = kp.dt;
  if (wid == 0) tm_alloc<ADJ_TM_COLS>(sm);
  __syncthreads();
  const uint32_t tm_base = *reinterpret_cast<volatile uint32_t*>(sm);
  const uint32_t tm = tm_base + (uint32_t(wid) << 21);  // warp w reaches the lanes 32 w ..
  static_assert(NT == 128, "a warp per quarter of the tensor memory's lanes");
  __syncthreads();

  for (int tix = blockIdx.x; tix < kp.n_tiles; tix += gridDim.x) {
    const Tile tile = kp.tiles[tix];
    const DevMember& M = kp.members[tile.member];
    const GitmColumnAdjoint B = (kp.n_inline > 0) ? kp.bars_inline[tile.member] : kp.bars[tile.member];
    const GitmColumnBatch& b = M.b;
    const int nA = (NA > 0) ? NA : b.n_alts;
    const int nc = tile.nc;
    const AdjLayout A = make_adj_layout(nA);
    const Layout& L = A.L;
    const int G = L.G;
    const int per = adj_state_doubles(nA);
    const int64_t ncols = b.n_cols;
    double* const eb = sm + size_t(A.stride) * nc;  // [ADJ_EDGE_DOUBLES]
    uint32_t* sst = reinterpret_cast<uint32_t*>(eb + ADJ_EDGE_DOUBLES);
    uint32_t* sfrozen = sst + nc;
    const int nitems = nc * nA;
    const bool item = tid < nitems;
    const bool wact = wid * 32 < nitems;  // warps with items run whole: the idle lanes of the last repeat its last item
    const int it = min(tid, nitems - 1);
    const int my_cl = it / nA;
    const int my_i = it % nA + 1;
    // the stage adjoint's neighbours of this thread's cell (cells of a
    // column are consecutive threads)
    const int nbl = !item ? NB_LANE : (my_i == 1) ? NB_GHOST : (lane == 0) ? NB_WARP : NB_LANE;
    const int nbr = !item ? NB_LANE : (my_i == nA) ? NB_GHOST : (lane == 31) ? NB_WARP : NB_LANE;

    auto ctx = [&](int cl) {
      ColCtx c;
      c.col = sm + size_t(A.stride) * cl;
      c.L = L;
      c.gridc = M.gridc;
      c.gcols = M.gcols;
      c.gc = (M.gcols == 1) ? 0 : int(tile.c0 + cl);
      c.xo = L.X0;
      c.xpo = L.XP0;
      return c;
    };
    auto adj = [&](int cl) {
      ColAdj a;
      double* col = sm + size_t(A.stride) * cl;
      a.xb = col + L.X1;
      a.xbp = col + L.XP1;
      a.db = col + A.DB;
      a.gu = col + A.GU;
      a.fb = col + A.FB;
      a.cmb = col + A.CMB;
      a.gmb = col + A.GMB;
      a.tub = col + A.TUB;
      a.mmb = col + A.MMB;
      a.lc = reinterpret_cast<uint8_t*>(col + A.LC);
      a.G = G;
      a.nA = nA;
      a.act = item;
      a.nbl = nbl;
      a.nbr = nbr;
      a.eb = eb;
      a.wid = wid;
      return a;
    };
    auto gidx = [&](int f, int g, int cl) -> int64_t { return (int64_t(f) * G + g) * ncols + tile.c0 + cl; };
    auto state = [&](int s, int cl) -> const double* {
      return kp.saved + (int64_t(s) * kp.saved_ncols + M.col_offset + tile.c0 + cl - kp.saved_c0) * kp.per_max;
    };
    // (the caller's barrier publishes the copies)
    auto load = [&](int s, int off) {
      for (int cl = 0; cl < nc; ++cl) {
        const double* src = state(s, cl);
        double* dst = sm + size_t(A.stride) * cl + off;
        for (int r = tid; r < per; r += NT) cp_async8(dst + r, src + r);
      }
      cp_async_wait_all();
    };
    // the thread's q-th ghost or passive-ion cell of the state adjoint (null: none)
    const int nog = (nc * ADJ_OG + NT - 1) / NT;
    auto ghost = [&](int q) -> double* {
      const int e = tid + q * NT, cl = e / ADJ_OG, r = e - cl * ADJ_OG;
      if (cl >= nc) return nullptr;
      const int u = r & 3;
      return sm + size_t(A.stride) * cl + L.X1 +
             (r < NF * 4 ? (r >> 2) * G + (u < 2 ? u : nA + u) : NF * G + r - NF * 4);
    };
    // bc^T of every column on the state in X0 (pg1, pg2: the pre-boundary ions
    // of this thread's column at nAlts+1 and nAlts+2): the ions of a column, the neutrals of two,
    // each a warp's task; the two ends of a column in turn where they meet
    auto boundaries_adjoint = [&](double pg1, double pg2) {
      const int np = (nc + 1) / 2;  // pairs of columns (nc <= nw: the ions are a warp's first task)
      const int ends = (nA >= 10) ? 2 : 1;
      for (int t = wid; t < nc + ends * np; t += nw) {
        if (t < nc) {
          bc_adjoint_ions(ctx(t), adj(t), pg1, pg2, prm, lane, &sst[t]);
        } else {
          const int p = (t - nc) % np, end = (t - nc) / np;
          const int cl = min(2 * p + (lane >> 4), nc - 1);
          const int s = (2 * p + (lane >> 4) < nc) ? lane & 15 : 15;
          if (end == 0) bc_adjoint_upper(ctx(cl), adj(cl), s);
          if (end == ends - 1) bc_adjoint_lower(ctx(cl), adj(cl), prm, s);
        }
      }
    };

    if (tid < nc) {
      sst[tid] = 0u;
      sfrozen[tid] = 0u;
    }
    __syncthreads();

    // ------------------------------------------------------------ gather
    // the column scalars and coefficients, as the forward kernel's load; the
    // state itself comes from the saved stage states
    if (tid < nc) {
      ColCtx c = ctx(tid);
      const int64_t cc = tile.c0 + tid;
      const double cl = b.cos_lat[cc];
      const double cent = (cl * prm.omega_body) * (cl * prm.omega_body);
      c.sc(SC_CENT) = cent;
      c.sc(SC_CORI) = 2 * cl * prm.omega_body;
      const double sza = b.sza[cc], mlat = b.mlat[cc];
      c.sc(SC_SZA) = sza;
      c.sc(SC_MLAT) = mlat;
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
    }
    for (int w = tid; w < nc * G; w += NT) {
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
        double N = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) N = N + nd[s];
        double gg = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) gg = gg + nd[s] * c_k.inv_vib2[s];
        gamma = gg * 2.0 / N + 1;
        double m = 0.0;
        const double rn = 1.0 / (N + 1.0);
#pragma unroll
        for (int s = 0; s < NS; ++s) m = m + c_k.mass[s] * nd[s] * rn;
        if (m == 0) m = c_k.mass[0];
        mmm = m;
        tu = m * (1.0 / KB);
        if (g >= 1 && g <= nA + 2) {
          double mx = fabs(ww[0]);
#pragma unroll
          for (int s = 1; s < NS; ++s) mx = fmax(mx, fabs(ww[s]));
          cmx = mx + sqrt(gamma * temperature);
        }
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
    }
    __syncthreads();  // @phase 0
    double eddy = 0.0, ivup = 0.0;
    if (item) {
      eddy = b.eddy[gidx(0, my_i + 1, my_cl)];
      ivup = b.ivel_up[gidx(0, my_i + 1, my_cl)];
    }
    // the pre-boundary ion ghosts of column `wid`, ion `lane`: Orig's and the gathered ones
    double pgx[2] = {0.0, 0.0}, pgo[2] = {0.0, 0.0};
    if (wid < nc && lane < NI) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = (lane < NADV) ? (F_I + lane) * G + nA + 2 + u : NF * G + (lane - NADV) * NPC + pcell(nA + 1 + u, nA);
        pgx[u] = state(1, wid)[r];
        pgo[u] = state(0, wid)[r];
      }
    }
    load(5, L.X0);  // X4
    __syncthreads();

    // ------------------------------------------------------------ reverse
    for (int cl = 0; cl < nc; ++cl) {
      double* col = sm + size_t(A.stride) * cl;
      for (int r = tid; r < per; r += NT) {
        col[L.X1 + r] = 0.0;
      }
      for (int r = A.DB + tid; r < A.stride; r += NT) col[r] = 0.0;
    }
    __syncthreads();  // @phase 0
    // scatter^T (advance_vertical.f90:163-217 and the heating line).  The
    // cell's output adjoints are read into registers first: read between
    // the shared-memory updates, each load would wait for the one before.
    for (int w = tid; w < nc * G; w += NT) {
      const int g = w / nc, cl = w - g * nc, i = g - 1;
      if (sfrozen[cl]) continue;
      const bool ions = prm.use_ion_advection != 0;
      const bool pc = in_pcells(i, nA);
      const bool interior = (i >= 1 && i <= nA);
      const double y_rho = B.rho[gidx(0, g, cl)];
      const double y_ve = B.velocity[gidx(0, g, cl)];
      const double y_vn = B.velocity[gidx(1, g, cl)];
      const double y_vu = B.velocity[gidx(2, g, cl)];
      const double ytemp = B.temperature[gidx(0, g, cl)];
      const bool heat = b.heating && interior && B.heating_scale;
      const double hq = heat ? b.heating[gidx(0, g, cl)] : 0.0;
      const double yN = B.ndensity ? B.ndensity[gidx(0, g, cl)] : 0.0;
      double y_w[NS], y_nd[NS], y_ln[NS], y_ion[NI];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        y_w[s] = B.vert_vel[gidx(s, g, cl)];
        y_nd[s] = B.ndensity_s[gidx(s, g, cl)];
        y_ln[s] = B.log_ns ? B.log_ns[gidx(s, g, cl)] : 0.0;
      }
      const double ye = ions ? B.idensity_s[gidx(NI, g, cl)] : 0.0;
#pragma unroll
      for (int s = 0; s < NI; ++s) y_ion[s] = (ions && (s < NADV || pc)) ? B.idensity_s[gidx(s, g, cl)] : 0.0;
      ColCtx c = ctx(cl);
      ColAdj a = adj(cl);
      const double tu = c.tu(i);
      const double LR4 = c.x(F_LRHO, i), T4 = c.x(F_T, i);
      a.x(F_LRHO, i) += y_rho * exp(LR4);
      a.x(F_VE, i) += y_ve;
      a.x(F_VN, i) += y_vn;
      a.x(F_VU, i) += y_vu;
      a.x(F_T, i) += ytemp / tu;
      a.tub[i + 1] += -(ytemp * T4 / tu) / tu;
      // the heating factor's adjoint of each interior cell, summed in cell
      // order below (GradLogConS's buffer is free until the stage adjoints)
      if (interior && b.heating && B.heating_scale) a.gu[i - 1] = heat ? ytemp * dt * hq : 0.0;
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        a.x(F_W + s, i) += y_w[s];
        const double L4 = c.x(F_LNS + s, i);
        double v = (y_nd[s] + yN) * exp(L4);
        if (B.log_ns) v += y_ln[s];
        a.x(F_LNS + s, i) += v;
      }
      if (ions) {
        const bool improved = prm.use_improved_ion_advection != 0;
#pragma unroll
        for (int s = 0; s < NI; ++s) {
          if (!(s < NADV || pc)) continue;
          const double I4 = c.ion(s, i);
          const double v = improved ? I4 : exp(I4);
          const bool floored = improved && interior && v < 1;
          const double yb = y_ion[s] + ye;
          a.ion(s, i) += floored ? 0.0 : (improved ? yb : yb * v);
        }
      }
    }
    __syncthreads();  // @phase 5
    if (tid < nc && !sfrozen[tid] && b.heating && B.heating_scale) {
      const double* hv = sm + size_t(A.stride) * tid + A.GU;
      double sum = 0.0;
      for (int i = 0; i < nA; ++i) sum += hv[i];
      sm[size_t(A.stride) * tid + A.MMB + 2] += sum;
    }
    double eddy_bar = 0.0;  // the four stages' KappaEddyDiffusion adjoints of this thread's cell
    // the boundary pass of the final state, then stage k and the boundary
    // pass of its state for k = 3 .. 0: one copy of each in the loop
#pragma unroll 1
    for (int k = 4;; --k) {
      if (k < 4) {
        load(1 + k, L.X0);
        for (int cl = 0; cl < nc; ++cl) {
          double* db = sm + size_t(A.stride) * cl + A.DB;
          for (int r = tid; r < NSTENCIL * (nA + 2); r += NT) db[r] = 0.0;
        }
        for (int r = tid; r < ADJ_EDGE_DOUBLES; r += NT) eb[r] = 0.0;
        __syncthreads();  // @phase 8
        for (int j = tid; j < nc * (nA + 2); j += NT) {
          const int cl = j / (nA + 2), i = j - cl * (nA + 2);
          slopes_with_branches(ctx(cl), adj(cl), i, prm.beta_limiter);
        }
        __syncthreads();  // @phase 8
        if (wact) {
          ColCtx c = ctx(my_cl);
          ColAdj a = adj(my_cl);
          eddy_bar += cell_adjoint_species(c, a, my_i, prm, dt, eddy, tm + ADJ_TM_K);
          cell_adjoint_rest(c, a, my_i, dt, ivup, tm + ADJ_TM_K);
        }
        __syncthreads();  // @phase 9
        // GradLogConS's shares of the neighbouring cells and the sweeps'
        // shares that crossed a warp boundary, one thread per cell
        for (int w = tid; w < nc * G; w += NT) {
          const int cl = w / G, m = w - cl * G - 1;
          cell_gather(ctx(cl), adj(cl), m, cl * nA, nitems);
        }
        // the other fields' edge shares and every slope's, a thread each (18
        // in turn by the two cells' threads took 5 kcycles)
        if (tid < (nw - 1) * NSTENCIL * 2) {
          const int side = tid & 1, f = (tid >> 1) % NSTENCIL, bnd = tid / (2 * NSTENCIL);
          const int t = edge_thread(bnd, side, nA, nitems);
          if (t >= 0) {
            const int cl = t / nA, i = t - cl * nA + 1;
            ColAdj a = adj(cl);
            const double* e = eb + (bnd * NSTENCIL + f) * 4 + 2 * side;
            if (f >= F_LNS + NS) a.x(f, i) += e[0];
            a.db[f * (nA + 2) + i] += e[1];
          }
        }
        __syncthreads();  // @phase 9
        {
          // (column, field, run of cells) per thread
          const int nseg = max(1, NT / (nc * NSTENCIL));
          const int seg = (G + nseg - 1) / nseg;
          for (int w = tid; w < nc * NSTENCIL * nseg; w += NT) {
            const int sg = w % nseg, r = w / nseg, f = r % NSTENCIL, cl = r / NSTENCIL;
            const int j0 = -1 + sg * seg, j1 = min(j0 + seg - 1, nA + 2);
            if (j0 <= j1) slopes_adjoint_run(ctx(cl), adj(cl), f, j0, j1, prm.beta_limiter);
          }
        }
        __syncthreads();  // @phase 10
        if (k == 0) {
          // X0 is also Orig
          if (wact) {
            ColAdj a = adj(my_cl);
#pragma unroll 1
            for (int f0 = 0; f0 < NF; f0 += 4) {
              double o[4];
              tm_get(tm + ADJ_TM_O + 2 * f0, o);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (j < 3 || f0 + 4 <= NF) a.own(f0 + j, my_i, o[j]);
            }
          }
          for (int q = 0; q < nog; ++q) {
            const double o = tm_get(tm + ADJ_TM_OG + 2 * q);
            if (double* p = ghost(q)) *p += o;
          }
          __syncthreads();  // @phase 7
        }
      }
      // pre-boundary ghosts: Orig's, the gathered ones for the first pass
      boundaries_adjoint(k > 0 ? pgx[0] : pgo[0], k > 0 ? pgx[1] : pgo[1]);
      __syncthreads();  // @phase 6
      if (k == 0) break;
      // combination^T: X4pre = Orig + (K0 + 2 K1 + 2 K2 + K3) / 6, Xkpre = Orig + c K(k-1), c = 1/2, 1/2, 1;
      // the state adjoint goes to Orig's and starts again from K = New - state's own -K
      if (wact) {
        ColAdj a = adj(my_cl);
        const double w = (k == 3 || k == 2) ? 2.0 : 1.0, cx = (k == 3) ? 1.0 : 0.5;
#pragma unroll 1
        for (int f0 = 0; f0 < NF; f0 += 4) {
          double kv[4], ac[4], o[4];
          const uint32_t at = tm + 2 * f0;
          if (k < 4) tm_get(at + ADJ_TM_K, at + ADJ_TM_ACC, at + ADJ_TM_O, kv, ac, o);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const bool on = j < 3 || f0 + 4 <= NF;
            const double x = on ? a.x(f0 + j, my_i) : 0.0;
            const double s = (1.0 / 6.0) * x;
            kv[j] = (k == 4) ? s : w * ac[j] + cx * x;
            ac[j] = (k == 4) ? s : ac[j];
            o[j] = (k == 4) ? x : o[j] + x;
            if (item && on) a.x(f0 + j, my_i) = -kv[j];
          }
          tm_put(at + ADJ_TM_K, kv);
          if (k == 4) tm_put(at + ADJ_TM_ACC, ac);
          tm_put(at + ADJ_TM_O, o);
        }
      }
      for (int q = 0; q < nog; ++q) {
        double* p = ghost(q);
        double o = p ? *p : 0.0;
        if (k < 4) o += tm_get(tm + ADJ_TM_OG + 2 * q);
        tm_put(tm + ADJ_TM_OG + 2 * q, o);
        if (p) *p = 0.0;
      }
      tm_put_wait();
      __syncthreads();  // @phase 7
    }

    if (item && B.eddy && !sfrozen[my_cl]) B.eddy[gidx(0, my_i + 1, my_cl)] += eddy_bar;

    // ------------------------------------------------------------ gather^T
    for (int w = tid; w < nc * G; w += NT) {
      const int g = w / nc, cl = w - g * nc, i = g - 1;
      if (sfrozen[cl]) continue;
      // every global value of the cell is read before its first global
      // store (a store could alias a later load, which would then wait)
      const bool ions = prm.use_ion_advection != 0;
      const bool pc = in_pcells(i, nA);
      double nd[NS], ww[NS], ndb[NS], wwb[NS], iv[NI];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        nd[s] = b.ndensity_s[gidx(s, g, cl)];
        ww[s] = b.vert_vel[gidx(s, g, cl)];
      }
      const double temperature = b.temperature[gidx(0, g, cl)];
      const double rho_in = b.rho[gidx(0, g, cl)];
      const double ye = ions ? B.idensity_s[gidx(NI, g, cl)] : 0.0;
#pragma unroll
      for (int s = 0; s < NI; ++s)
        iv[s] = !ions ? 0.0 : (s < NADV || pc) ? b.idensity_s[gidx(s, g, cl)] : B.idensity_s[gidx(s, g, cl)];
      ColCtx c = ctx(cl);
      ColAdj a = adj(cl);
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        ndb[s] = a.x(F_LNS + s, i) / nd[s];
        wwb[s] = a.x(F_W + s, i);
      }
      const double tu = c.tu(i);
      double tb = a.x(F_T, i) * tu;
      double tub = a.tub[i + 1] + a.x(F_T, i) * temperature;
      if (prm.compute_coefficients) {
        double N = 0.0, gg = 0.0, ms = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) N = N + nd[s];
#pragma unroll
        for (int s = 0; s < NS; ++s) gg = gg + nd[s] * c_k.inv_vib2[s];
        const double gamma = gg * 2.0 / N + 1;
        const double rn = 1.0 / (N + 1.0);
#pragma unroll
        for (int s = 0; s < NS; ++s) ms = ms + c_k.mass[s] * nd[s];
        double gammab = a.gmb[i + 1];
        if (g >= 1 && g <= nA + 2) {
          const double cb = a.cmb[i + 1];
          int am = 0;
          double mx = fabs(ww[0]);
#pragma unroll
          for (int s = 1; s < NS; ++s)
            if (fabs(ww[s]) > mx) {
              mx = fabs(ww[s]);
              am = s;
            }
          wwb[am] += cb * ((ww[am] < 0.0) ? -1.0 : (ww[am] > 0.0 ? 1.0 : 0.0));
          const double sq = sqrt(gamma * temperature);
          gammab += cb * temperature / (2.0 * sq);
          tb += cb * gamma / (2.0 * sq);
        }
        double mb = tub * (1.0 / KB);
        if (i == -1) mb += a.mmb[0];
        if (i == 0) mb += a.mmb[1];
        const double rnb = mb * ms;
        double Nb = rnb * (-rn * rn);
        const double ggb = gammab * 2.0 / N;
        Nb += -gammab * gg * 2.0 / (N * N);
#pragma unroll
        for (int s = 0; s < NS; ++s) ndb[s] += mb * c_k.mass[s] * rn + ggb * c_k.inv_vib2[s] + Nb;
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        B.ndensity_s[gidx(s, g, cl)] = ndb[s];
        B.vert_vel[gidx(s, g, cl)] = wwb[s];
      }
      B.temperature[gidx(0, g, cl)] = tb;
      B.velocity[gidx(0, g, cl)] = a.x(F_VE, i);
      B.velocity[gidx(1, g, cl)] = a.x(F_VN, i);
      B.velocity[gidx(2, g, cl)] = a.x(F_VU, i);
      B.rho[gidx(0, g, cl)] = a.x(F_LRHO, i) / rho_in;
      if (ions) {
        const bool improved = prm.use_improved_ion_advection != 0;
#pragma unroll
        for (int s = 0; s < NI; ++s) {
          // advected ions: the state value iv; the others: their own
          // output adjoint iv, unchanged by the step, summed into e-
          if (s < NADV || pc)
            B.idensity_s[gidx(s, g, cl)] = improved ? a.ion(s, i) : a.ion(s, i) / iv[s];
          else
            B.idensity_s[gidx(s, g, cl)] = iv[s] + ye;
        }
        B.idensity_s[gidx(NI, g, cl)] = 0.0;
      }
    }
    if (tid < nc && !sfrozen[tid] && b.heating && B.heating_scale)
      B.heating_scale[tile.c0 + tid] += sm[size_t(A.stride) * tid + A.MMB + 2];
    if (tid < nc) {
      const int64_t gcol = M.col_offset + tile.c0 + tid;
      uint32_t wv = sst[tid];
      if (sfrozen[tid]) wv |= GITM_ST_NEG_DENSITY;
      if (wv) kp.status[gcol] |= wv;
    }
    __syncthreads();  // @phase 11
  }
  if (wid == 0) tm_free<ADJ_TM_COLS>(tm_base);
}

}  // namespace gv
