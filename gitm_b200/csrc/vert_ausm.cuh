// vert_ausm.cuh -- the AUSM stage of the vertical step (UseAUSMSolver), run
// by vert_step_kernel when the solver is GITM_SOLVER_AUSM.
//
// advance_vertical_1stage_ausm (vertical_solver_ausm.f90:436-999) with the
// AUSM+-up fluxes of calc_all_fluxes_hydro (:1093-2070) at both faces of the
// thread's cell.  Layout of the slope buffer (L.DL, 32 fields):
//   0..5   LogRhoS   (2nd-order "kt" slopes, calc_kt_facevalues :2073-2117)
//   6..11  LogPS     (kt)
//   12..17 LogHydroPressureS (kt)
//   18..23 VertVel   (kt)
//   24,25  Vel east / north (kt)
//   26     Gamma     (kt)
//   27     Temp      (4th-order slopes, calc_facevalues_alts_ausm)
//   28,29  Vel east / north (4th order)
//   30,31  ions 1, 2 (4th order, calc_rusanov_alts_rusanov)
// Values are formed in log space where the reference multiplies and takes
// the log: LogRhoS = log m + LogNS, LogPS = LogNS + log k + log T, and the
// hydrostatic species pressure (:714-751) is
//   log HydroPressureS(i) = LogNS(0) + log k + log T(0) + m_s Q(i),
//   Q(i) = sum_{j=1..i} dAlt_F(j) MeanGravity(j) / (k MeanTemp(j)),
// because the temperature ratios of the upward recurrence telescope.
#pragma once

namespace gv {

enum AusmSlope : int {
  AS_LRHOS = 0, AS_LPS = 6, AS_LHPS = 12, AS_W = 18, AS_VE = 24, AS_VN = 25, AS_GAM = 26,
  AS_T4 = 27, AS_VE4 = 28, AS_VN4 = 29, AS_I4 = 30
};
constexpr int SC_QB = 59;  // dAlt_F(-1) * InvScaleHeight of the bulk gas below cell 0

__device__ __forceinline__ double sqr(double x) { return x * x; }

// log HydroPressureS(i) - (LogNS(0) + log k + log T(0)) for species s
__device__ __forceinline__ double hydro_q(ColCtx c, int s, int i) {
  return (i < 0) ? c.sc(SC_QB) : c_k.mass[s] * c.col[c.L.QS + i + 1];
}

// the value of AUSM slope field f at cell i
__device__ __forceinline__ double ausm_field(ColCtx c, int f, int i) {
  if (f < AS_LPS) return c.x(F_LNS + f, i);  // LogRhoS - log m
  if (f < AS_LHPS) return c.x(F_LNS + f - AS_LPS, i) + c.col[c.L.LT + i + 1];  // LogPS - log k
  if (f < AS_W) return hydro_q(c, f - AS_LHPS, i);  // LogHPS - base
  if (f < AS_VE) return c.x(F_W + f - AS_W, i);
  if (f == AS_VE || f == AS_VE4) return c.x(F_VE, i);
  if (f == AS_VN || f == AS_VN4) return c.x(F_VN, i);
  if (f == AS_GAM) return c.gm(i);
  if (f == AS_T4) return c.x(F_T, i);
  return c.x(F_I + f - AS_I4, i);
}

// Phase A1: log T on every cell, and the prefix sum Q (one warp per column).
__device__ __forceinline__ void ausm_prefix(ColCtx c, int lane) {
  const int nA = c.L.nAlts;
  double* Q = c.col + c.L.QS + 1;  // Q[i]
  double carry = 0.0;
  if (lane == 0) Q[0] = 0.0;
  for (int base = 1; base <= nA + 2; base += 32) {
    const int j = base + lane;
    double t = 0.0;
    if (j <= nA + 2) {
      const double mg = 0.5 * (c.g(GC_GRAV, j) + c.sc(SC_CENT) * c.g(GC_R, j) + c.g(GC_GRAV, j - 1) +
                               c.sc(SC_CENT) * c.g(GC_R, j - 1));
      const double mt = 0.5 * (c.x(F_T, j) + c.x(F_T, j - 1));
      t = c.dAF(j) * mg / (KB * mt);
    }
    for (int off = 1; off < 32; off <<= 1) {
      const double u = __shfl_up_sync(0xffffffffu, t, off);
      if (lane >= off) t += u;
    }
    if (j <= nA + 2) Q[j] = carry + t;
    carry += __shfl_sync(0xffffffffu, t, 31);
  }
  if (lane == 0) {
    // cell -1 from cell 0 with the mean major mass (:734-742)
    const double MeanMass = 0.5 * (c.sc(SC_MMM_M1) + c.sc(SC_MMM_0));
    const double MeanGravity = 0.5 * (c.sc(SC_EG + 1) + c.sc(SC_EG + 0));
    const double MeanTemp = 0.5 * (c.x(F_T, 0) + c.x(F_T, -1));
    const double ish = -1.0 * MeanMass * MeanGravity / (KB * MeanTemp);
    c.sc(SC_QB) = c.dAF(-1) * ish;
  }
}

// Phase A2: the 32 slopes at cell i (0..nAlts+1): 2nd-order "kt" slopes, and
// the 4th-order form of the last five (2nd-order at cells 0 and nAlts+1).  A
// species' values are read once for its density and pressure slopes, and the
// grid's coefficients once for all, ahead of the stores they would otherwise
// be read again after (2.5 degrees, 4 steps: 6.94 -> 5.96 ms; 6.09 with the
// warps brought together at every tensor-memory access).
__device__ __forceinline__ void ausm_slopes_cell(ColCtx c, int i, double beta) {
  const int nA = c.L.nAlts;
  const double id1 = c.g(GC_IDF, i + 1), id0 = c.g(GC_IDF, i);
  const bool end = i == 0 || i == nA + 1;
  const double h1 = end ? 0.0 : c.g(GC_H2, i + 1), h0 = end ? 0.0 : c.g(GC_H2, i);
  double* const sl = &c.dl(0, i);
  const int pd = c.L.PD;
  auto kt = [&](double vm, double v0, double vp) { return limiter_mc((vp - v0) * id1, (v0 - vm) * id0, beta); };
  const double* lt = c.col + c.L.LT + i + 1;
  const double* q = c.col + c.L.QS + i + 1;
  const double ltm = lt[-1], lt0 = lt[0], ltp = lt[1];
  const double qm = q[i > 0 ? -1 : 0], q0 = q[0], qp = q[1], qb = c.sc(SC_QB);
#pragma unroll 2
  for (int s = 0; s < NS; ++s) {
    const double lm = c.x(F_LNS + s, i - 1), l0 = c.x(F_LNS + s, i), lp = c.x(F_LNS + s, i + 1);
    const double wm = c.x(F_W + s, i - 1), w0 = c.x(F_W + s, i), wp = c.x(F_W + s, i + 1);
    const double m = c_k.mass[s];
    const double a = kt(lm, l0, lp), b = kt(lm + ltm, l0 + lt0, lp + ltp);
    const double h = kt(i > 0 ? m * qm : qb, m * q0, m * qp), w = kt(wm, w0, wp);
    sl[(AS_LRHOS + s) * pd] = a;
    sl[(AS_LPS + s) * pd] = b;
    sl[(AS_LHPS + s) * pd] = h;
    sl[(AS_W + s) * pd] = w;
  }
  sl[AS_GAM * pd] = kt(c.gm(i - 1), c.gm(i), c.gm(i + 1));
  const int ip2 = min(i + 2, nA + 2), im2 = max(i - 2, -1);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int f = k == 0 ? F_T : k < 3 ? F_VE + k - 1 : F_I + k - 3;
    const double vmm = c.x(f, im2), vm = c.x(f, i - 1), v0 = c.x(f, i), vp = c.x(f, i + 1), vpp = c.x(f, ip2);
    const double u2 = (vp - v0) * id1, d2 = (v0 - vm) * id0;
    const double u4 = h1 * (0.6250000 * (vp - v0) - 0.0416667 * (vpp - vm));
    const double d4 = h0 * (0.6250000 * (v0 - vm) - 0.0416667 * (vp - vmm));
    if (k == 1 || k == 2) sl[(AS_VE + k - 1) * pd] = limiter_mc(u2, d2, beta);
    sl[(AS_T4 + k) * pd] = limiter_mc(end ? u2 : u4, end ? d2 : d4, beta);
  }
  static_assert(AS_VE4 == AS_T4 + 1 && AS_VN4 == AS_T4 + 2 && AS_I4 == AS_T4 + 3 && F_VN == F_VE + 1, "the order of the fields");
}

// kt face values of a field at the lower (M) and upper (P) faces of cell i:
// left/right states (calc_kt_facevalues :2105-2111)
struct Faces {
  double lm, rm, lp, rp;
};
__device__ __forceinline__ Faces kt_faces(ColCtx c, int f, int i, double vm, double v0, double vp) {
  const double* d = &c.col[c.L.DL + f * (c.L.nAlts + 2)];
  // halves of the cell widths: a product with 0.5 is exact, so d * (0.5 dF)
  // rounds like (0.5 d) dF
  const double hm = 0.5 * c.dAF(i - 1), h0 = 0.5 * c.dAF(i), hp = 0.5 * c.dAF(i + 1);
  Faces r;
  r.lm = fma(d[i - 1], hm, vm);
  r.rm = fma(-d[i], h0, v0);
  r.lp = fma(d[i], h0, v0);
  r.rp = fma(-d[i + 1], hp, vp);
  return r;
}

// Rusanov gradient and dissipation from the 4th-order slopes (calc_rusanov_alts_*)
__device__ __forceinline__ void ausm_sweep(ColCtx c, int fslope, int ffield, int i, double fc0,
                                           double fc1, double& grad, double& diff) {
  const double* v = &c.col[c.xo + ffield * c.L.G + 1];
  const double* d = &c.col[c.L.DL + fslope * (c.L.nAlts + 2)];
  const double hF0 = 0.5 * c.dAF(i), hF1 = 0.5 * c.dAF(i + 1), idc = c.g(GC_IDC, i);
  const double L0 = fma(d[i - 1], hF0, v[i - 1]);
  const double R0 = fma(-d[i], hF0, v[i]);
  const double L1 = fma(d[i], hF1, v[i]);
  const double R1 = fma(-d[i + 1], hF1, v[i + 1]);
  grad = (L1 + R1 - L0 - R0) * (0.5 * idc);
  diff = (fc1 * (R1 - L1) - fc0 * (R0 - L0)) * idc;
}

// exp of the four face states of a field shifted by `base`.
__device__ __forceinline__ void exp_faces(const Faces& t, double base, double (&e)[4]) {
  const double a[4] = {base + t.lm, base + t.rm, base + t.lp, base + t.rp};
  exp_n(a, e);
}

// AUSM+-up numerical velocity (Mach split, pressure diffusion) at one face
// and the species flux pair; (:1660-1937).  ics = 1 / cs; kp = LiouKpS times
// MPRESS_SCALE, which with the mean density's keeps the pressure diffusion's
// denominator a normal number for a species of hardly any density (both
// products are exact).
constexpr double MPRESS_SCALE = 0x1p64;
__device__ __forceinline__ void species_face_flux(double rl, double rr, double pl, double pr, double hl,
                                                  double hr, double wl, double wr, double cs, double ics, double kp,
                                                  double ku, double dzdt, bool subtract, double& nv,
                                                  double& rflux, double& mflux, double& np) {
  const double MInf = 1.0e-19;
  const double Ml = wl * ics, Mr = wr * ics;
  const double Ml2 = sqr(Ml), Mr2 = sqr(Mr);
  const double M2Bar = 0.5 * (Ml2 + Mr2);
  const double M2Zero = fmin(1.0, fmax(M2Bar, MInf));
  const double MZero = sqrt(M2Zero);
  const double FA = MZero * (2.0 - MZero);
  // MF4P(Ml) + MF4N(Mr) of :1700-1760 with LiouBeta = 1/8.  For |M| < 1 the
  // products multiply out to 3/8 + M/2 + M^4/8 and -3/8 + M/2 - M^4/8: the
  // constants cancel before the sum instead of in it (winds are 1e-2 of the
  // sound speed and less).  For |M| >= 1: (M + |M|) / 2 and (M - |M|) / 2.
  const double FL = (fabs(Ml) >= 1.0) ? 0.5 * (Ml + fabs(Ml)) - 0.375 : fma(0.125 * Ml2, Ml2, 0.5 * Ml);
  const double FR = (fabs(Mr) >= 1.0) ? 0.5 * (Mr - fabs(Mr)) + 0.375 : fma(-0.125 * Mr2, Mr2, 0.5 * Mr);
  const double meanrho = (0.5 * MPRESS_SCALE) * (rl + rr);
  const double dp = subtract ? ((pr - hr) - (pl - hl)) : (pr - pl);
  const double MPress = kp * fmax(1.0 - M2Bar, 0.0) * dp * rcp_nr(meanrho * cs * (FA * cs + 1.0 * dzdt));
  nv = cs * (FL + FR - MPress);
  const double meanp = 0.5 * (pl + pr);
  const double base = subtract ? (meanp - 0.5 * (hl + hr)) : meanp;
  np = base - 0.5 * ku * cs * (rr * wr - rl * wl);
  const bool up = nv >= 0.0;
  rflux = (up ? rl : rr) * nv;
  mflux = (up ? rl * wl : rr * wr) * nv;
}

constexpr uint32_t AUSM_TM_ND = 136;

// advance_vertical_1stage_ausm (vertical_solver_ausm.f90:436-999) at interior
// cell i with stage step dtk; emit(f, New - state) takes each new value.
// The face fluxes of calc_all_fluxes_hydro are formed at the cell's two
// faces in two passes over the species: the first sums the bulk face states
// (densities, pressures, mass-weighted vertical wind), which set the Liou
// sound speed; the second forms the species fluxes and applies them.
// TM: the first pass's face states are kept in the thread's tensor memory
// (NS x 16 columns at tm) for the second, which leaves its results there; the
// cell's densities and deviations at tm + AUSM_TM_ND, 4 columns a species.
// Whole warps call.
template <bool TM, class Emit>
__device__ __forceinline__ void ausm_cell(ColCtx c, int i, const GitmVertParams& prm, double dtk,
                                          double eddy, double ivup, uint32_t tm, Emit&& emit,
                                          uint32_t* st = nullptr) {
  const int nA = c.L.nAlts;
  (void)nA;
  const double logk = c_k.log_kb;
  const double T = c.x(F_T, i), VE = c.x(F_VE, i), VN = c.x(F_VN, i), VU = c.x(F_VU, i);
  const double LR = c.x(F_LRHO, i);
  const double EG = c.g(GC_GRAV, i) + c.sc(SC_CENT) * c.g(GC_R, i);
  const double invr = c.g(GC_INVR, i);
  const double gam = c.gm(i);

  // Rusanov sweeps whose results the stage reads (:580-640)
  const double fc0 = 0.5 * fmax(c.cm(i - 1), c.cm(i));
  const double fc1 = 0.5 * fmax(c.cm(i), c.cm(i + 1));
  double gT, dT, gE, dE, gN, dN;
  ausm_sweep(c, AS_T4, F_T, i, fc0, fc1, gT, dT);
  ausm_sweep(c, AS_VE4, F_VE, i, fc0, fc1, gE, dE);
  ausm_sweep(c, AS_VN4, F_VN, i, fc0, fc1, gN, dN);
  (void)gE;
  (void)gN;

  // cell values (:560-575, 752-790)
  double ns[NS], Rho;
  double NT = 0.0;
  {
    double l[NS + 1], e[NS + 1];
#pragma unroll
    for (int s = 0; s < NS; ++s) l[s] = c.x(F_LNS + s, i);
    l[NS] = LR;
    exp_n(l, e);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      ns[s] = e[s];
      NT = NT + ns[s];
    }
    Rho = e[NS];
  }
  const double Press = NT * KB * T;
  const double TotalEnergy = Press / (gam - 1.0) + 0.5 * Rho * (VU * VU + VN * VN + VE * VE);
  const double MomE = Rho * VE, MomN = Rho * VN;
  // hydrostatic species densities relative to the cell (:714-790):
  // log HydroNS(i) = LogNS(0) + log T(0) - log T(i) + m_s Q(i)
  const double lt0 = c.col[c.L.LT + 1], lti = c.col[c.L.LT + i + 1];
  unsigned sub = 0;  // SubtractHydrostatic bits
  double dev[NS];
  {
    double l[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) l[s] = c.x(F_LNS + s, 0) + lt0 - lti + hydro_q(c, s, i);
    exp_n(l, dev);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double RhoS = c_k.mass[s] * ns[s];
      dev[s] = RhoS - c_k.mass[s] * dev[s];
      if (!(fabs(dev[s]) > RhoS)) sub |= 1u << s;  // |RhoS - HydroRhoS| / RhoS > 1
    }
  }

  if constexpr (TM) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      tm_put(tm + AUSM_TM_ND + 4 * s, ns[s]);
      tm_put(tm + AUSM_TM_ND + 4 * s + 2, dev[s]);
    }
  }

  // ---- pass 1: bulk face states
  double RhoLM = 0.0, RhoRM = 0.0, RhoLP = 0.0, RhoRP = 0.0;
  double PLM = 0.0, PRM = 0.0, PLP = 0.0, PRP = 0.0;
  double WLM = 0.0, WRM = 0.0, WLP = 0.0, WRP = 0.0;  // sums of RhoS * VertVel
  // one species at a time: the fully unrolled passes made a body the
  // instruction cache could not hold.  The faces' exponentials go in batches
  // and the divisions that a face's species share are taken once; with one
  // copy of the boundary passes in the kernel (409 -> 238 KB of code) 2.5
  // degrees, 4 steps: 10.5 -> 8.5 ms; with the face states, the loop's values,
  // K and the accumulators in tensor memory (TM) 6.9 ms
  // the density and pressure face states of each species, kept from this
  // pass for the flux pass (without TM in per-thread memory)
  double fst[TM ? 1 : NS][8];
#pragma unroll 1
  for (int s = 0; s < NS; ++s) {
    const double lm = c_k.log_mass[s];
    const Faces tr = kt_faces(c, AS_LRHOS + s, i, c.x(F_LNS + s, i - 1), c.x(F_LNS + s, i), c.x(F_LNS + s, i + 1));
    const Faces tp = kt_faces(c, AS_LPS + s, i, ausm_field(c, AS_LPS + s, i - 1), ausm_field(c, AS_LPS + s, i),
                              ausm_field(c, AS_LPS + s, i + 1));
    const Faces w = kt_faces(c, AS_W + s, i, c.x(F_W + s, i - 1), c.x(F_W + s, i), c.x(F_W + s, i + 1));
    const double a[8] = {lm + tr.lm,   lm + tr.rm,   lm + tr.lp,   lm + tr.rp,
                         logk + tp.lm, logk + tp.rm, logk + tp.lp, logk + tp.rp};
    double e[8];
    exp_n(a, e);
    if constexpr (TM) {
      __syncwarp();
      tm_put(tm + 16 * s, e);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) fst[s][j] = e[j];
    }
    RhoLM = RhoLM + e[0];
    RhoRM = RhoRM + e[1];
    RhoLP = RhoLP + e[2];
    RhoRP = RhoRP + e[3];
    PLM = PLM + e[4];
    PRM = PRM + e[5];
    PLP = PLP + e[6];
    PRP = PRP + e[7];
    WLM = WLM + e[0] * w.lm;
    WRM = WRM + e[1] * w.rm;
    WLP = WLP + e[2] * w.lp;
    WRP = WRP + e[3] * w.rp;
  }
  if constexpr (TM) tm_put_wait();
  // bulk face winds (:1503-1530): the up component is the mass-weighted species wind
  const double ULM = WLM / RhoLM, URM = WRM / RhoRM, ULP = WLP / RhoLP, URP = WRP / RhoRP;
  const Faces fE = kt_faces(c, AS_VE, i, c.x(F_VE, i - 1), VE, c.x(F_VE, i + 1));
  const Faces fN = kt_faces(c, AS_VN, i, c.x(F_VN, i - 1), VN, c.x(F_VN, i + 1));
  const Faces fG = kt_faces(c, AS_GAM, i, c.gm(i - 1), gam, c.gm(i + 1));
  // energies, enthalpies (:1533-1565) and the Liou interface sound speed (:1568-1655)
  auto ke = [](double u, double e, double n) { return u * u + e * e + n * n; };
  const double KLM = ke(ULM, fE.lm, fN.lm), KRM = ke(URM, fE.rm, fN.rm);
  const double KLP = ke(ULP, fE.lp, fN.lp), KRP = ke(URP, fE.rp, fN.rp);
  auto enthalpy = [](double g, double P, double rho, double k2) { return 0.5 * k2 + (g / (g - 1.0)) * P / rho; };
  auto csound = [](double g, double H) { return sqrt(2.0 * ((g - 1.0) / (g + 1.0)) * H); };
  double CSM, CSP;
  {
    const double sl = csound(fG.lm, enthalpy(fG.lm, PLM, RhoLM, KLM));
    const double sr = csound(fG.rm, enthalpy(fG.rm, PRM, RhoRM, KRM));
    CSM = fmin(sqr(sl) / fmax(sl, ULM), sqr(sr) / fmax(sr, -1.0 * URM));
  }
  {
    const double sl = csound(fG.lp, enthalpy(fG.lp, PLP, RhoLP, KLP));
    const double sr = csound(fG.rp, enthalpy(fG.rp, PRP, RhoRP, KRP));
    CSP = fmin(sqr(sl) / fmax(sl, ULP), sqr(sr) / fmax(sr, -1.0 * URP));
  }

  // ---- pass 2: species fluxes, continuity and species momentum (:844-900)
  const double AP = c.ga(GA_AP, i), AM = c.ga(GA_AM, i), Vol = c.ga(GA_VOL, i);
  const double dAltC = c.ga(GA_DALTC, i);
  const double kp = MPRESS_SCALE * c.ga(GA_KP, i), ku = c.ga(GA_KU, i);
  const double dzdt = dAltC / dtk;
  const double hz = dtk * (VN * VN + VE * VE) * invr;
  const double iCSM = rcp_nr(CSM), iCSP = rcp_nr(CSP), iVol = rcp_nr(Vol), idAltC = rcp_nr(dAltC);
  double BulkVM = 0.0, BulkVP = 0.0;
  double nrs[NS], wv[NS];
  const double lnk0 = logk + c.col[c.L.LT + 1];  // log k + log T(0)
#pragma unroll 1
  for (int s = 0; s < NS; ++s) {
    const bool sh = (sub >> s) & 1u;
    double h[4] = {0.0, 0.0, 0.0, 0.0};
    if (sh)
      exp_faces(kt_faces(c, AS_LHPS + s, i, hydro_q(c, s, i - 1), hydro_q(c, s, i), hydro_q(c, s, i + 1)),
                c.x(F_LNS + s, 0) + lnk0, h);
    const Faces w = kt_faces(c, AS_W + s, i, c.x(F_W + s, i - 1), c.x(F_W + s, i), c.x(F_W + s, i + 1));
    double f[8], nd[4];
    if constexpr (TM) {
      __syncwarp();
      tm_get(tm + 16 * s, f);
      tm_get(tm + AUSM_TM_ND + 4 * s, nd);
    } else {
      nd[0] = ns[s];
      nd[1] = dev[s];
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = fst[s][j];
    }
    double nvM, rfM, mfM, npM, nvP, rfP, mfP, npP;
    species_face_flux(f[0], f[1], f[4], f[5], h[0], h[1], w.lm, w.rm, CSM, iCSM, kp, ku, dzdt, sh, nvM, rfM, mfM, npM);
    species_face_flux(f[2], f[3], f[6], f[7], h[2], h[3], w.lp, w.rp, CSP, iCSP, kp, ku, dzdt, sh, nvP, rfP, mfP, npP);
    BulkVP = BulkVP + (f[2] + f[3]) * nvP;
    BulkVM = BulkVM + (f[0] + f[1]) * nvM;
    const double RhoSFlux = (AP * rfP - AM * rfM) * iVol;
    const double MomSFlux = (AP * mfP - AM * mfM) * iVol + (npP - npM) * idAltC;
    const double RhoS = c_k.mass[s] * nd[0];
    const double Ws = c.x(F_W + s, i);
    const double NewRhoS = RhoS - dtk * RhoSFlux;
    const double MomS = RhoS * Ws;
    const double NewMomS = MomS - dtk * MomSFlux + dtk * (sh ? nd[1] : RhoS) * EG;
    double w1 = NewMomS / NewRhoS;
    w1 = w1 + hz;
    if (prm.use_coriolis) w1 = w1 + dtk * (c.sc(SC_CORI) * VE);
    w1 = w1 - dtk * (prm.thermal_diff_coef[s] * c_k.k_over_m[s]) * gT;
    if constexpr (TM) {
      const double r[4] = {NewRhoS, w1, 0.0, 0.0};
      __syncwarp();
      tm_put(tm + 16 * s, r);
    } else {
      nrs[s] = NewRhoS;
      wv[s] = w1;
    }
  }
  if constexpr (TM) {
    static_assert(NS == 6, "two groups of three species");
    tm_put_wait();
#pragma unroll
    for (int s = 0; s < NS; s += 3) {
      double u[4], v[4], w[4];
      tm_get(tm + 16 * s, tm + 16 * s + 16, tm + 16 * s + 32, u, v, w);
      nrs[s] = u[0];
      nrs[s + 1] = v[0];
      nrs[s + 2] = w[0];
      wv[s] = u[1];
      wv[s + 1] = v[1];
      wv[s + 2] = w[1];
    }
  }
  BulkVP = BulkVP / (RhoLP + RhoRP);
  BulkVM = BulkVM / (RhoLM + RhoRM);
  double NewRho = 0.0, NewNT = 0.0, nns[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    // nrs / mass, the product with the reciprocal corrected by its residual
    const double q = nrs[s] * c_k.inv_mass[s];
    nns[s] = fma(fma(-q, c_k.mass[s], nrs[s]), c_k.inv_mass[s], q);
    NewRho = NewRho + nrs[s];
    NewNT = NewNT + nns[s];
  }
  {
    // New LogNS and New LogRho (:993-996)
    double r[NS + 1], l[NS + 1];
#pragma unroll
    for (int s = 0; s < NS; ++s) r[s] = nns[s];
    r[NS] = NewRho;
    log_n(r, l);
#pragma unroll
    for (int s = 0; s < NS; ++s) emit(F_LNS + s, l[s] - c.x(F_LNS + s, i));
    emit(F_LRHO, l[NS] - LR);
  }
  const double iNewRho = 1.0 / NewRho;
  // friction on the updated densities with the stage temperature (:902-913)
  if (prm.use_neutral_friction) {
    friction_solve(dtk, nns, nrs, T, wv, st);
    if (eddy != 0.0) {
      double glc[NS];
      grad_log_cons(c, i, glc);
#pragma unroll
      for (int s = 0; s < NS; ++s) wv[s] = fma(-eddy, glc[s], wv[s]);
    }
  }
  // clamp and bulk vertical wind (:916-941)
  double NewVU = 0.0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    double w = (wv[s] > -prm.max_vertical_velocity) ? wv[s] : -prm.max_vertical_velocity;
    w = (w < prm.max_vertical_velocity) ? w : prm.max_vertical_velocity;
    emit(F_W + s, w - c.x(F_W + s, i));
    NewVU = NewVU + w * nrs[s];
  }
  NewVU = NewVU * iNewRho;
  emit(F_VU, NewVU - VU);

  // bulk energy and horizontal momentum fluxes (:1960-2026, 2041-2068)
  auto bulk = [&](bool left, double gl, double gr, double Pl, double Pr, double Rl, double Rr, double Kl, double Kr,
                  double el, double er, double nl, double nr, double V, double& EF, double& ME, double& MN) {
    const double g = left ? gl : gr, P = left ? Pl : Pr, R = left ? Rl : Rr, K = left ? Kl : Kr;
    EF = ((1.0 / (g - 1.0)) * P + 0.5 * R * K + P) * V;
    ME = R * (left ? el : er) * V;
    MN = R * (left ? nl : nr) * V;
  };
  double EFP, EFM, MEP, MEM, MNP, MNM;
  bulk(BulkVP >= 0.0, fG.lp, fG.rp, PLP, PRP, RhoLP, RhoRP, KLP, KRP, fE.lp, fE.rp, fN.lp, fN.rp, BulkVP, EFP, MEP, MNP);
  bulk(BulkVM >= 0.0, fG.lm, fG.rm, PLM, PRM, RhoLM, RhoRM, KLM, KRM, fE.lm, fE.rm, fN.lm, fN.rm, BulkVM, EFM, MEM, MNM);
  const double EnergyFlux = (AP * EFP - AM * EFM) * iVol;
  const double MomFluxE = (AP * MEP - AM * MEM) * iVol;
  const double MomFluxN = (AP * MNP - AM * MNM) * iVol;

  // horizontal winds, energy and temperature (:944-986)
  const double damp = c.ga(GA_DAMP, i);
  double NewVE = (MomE - dtk * MomFluxE) * iNewRho;
  NewVE = NewVE + damp * dtk * dE;
  double NewVN = (MomN - dtk * MomFluxN) * iNewRho;
  NewVN = NewVN + damp * dtk * dN;
  emit(F_VE, NewVE - VE);
  emit(F_VN, NewVN - VN);
  const double NewTotalEnergy = TotalEnergy - dtk * EnergyFlux + dtk * Rho * VU * EG;
  const double NewPress =
      (NewTotalEnergy - 0.5 * NewRho * (NewVU * NewVU + NewVN * NewVN + NewVE * NewVE)) * (gam - 1.0);
  emit(F_T, NewPress / (KB * NewNT) - T);

#pragma unroll
  for (int s = 0; s < NADV; ++s) {
    double gI, dI;
    ausm_sweep(c, AS_I4 + s, F_I + s, i, fc0, fc1, gI, dI);
    const double I = c.x(F_I + s, i);
    emit(F_I + s, (I - dtk * (ivup * gI) + dtk * dI) - I);  // :857-860
  }
}

}  // namespace gv
