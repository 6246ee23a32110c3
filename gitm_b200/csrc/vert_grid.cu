// vert_grid.cu -- grid coefficients of a plan, in the reference's operation
// order: dAlt_F / InvDAlt_F (advance_vertical.f90:149-151), the 5-point
// GradLogConS mesh (vertical_solver_rusanov.f90:515-533), the one-sided
// boundary meshes (set_vertical_bcs.Earth.f90:279-297, 505-525) and the AUSM
// cell constants (vertical_solver_ausm.f90:944-946, 1314-1352, 2029-2039).
//
// A thread per (cell, grid column); what bounds it is the write of 20 rows
// per cell.  GITM's own arrays hold an altitude grid per column, and one host
// thread took 20 ms for the 2,592 columns of a 5 degree globe, with a 23 MB
// upload; here 0.02 ms (the Fortran-array call of 32 blocks of
// 9 x 9 columns on the device: 22 -> 1.6 ms).  Compiled with -fmad=false (gitm_b200/build.py): sums
// and products round as the reference's, which uses no fused multiply-add.
#include "vert_grid.cuh"

namespace gv {

namespace {

constexpr int GRID_THREADS = 128;

__global__ void __launch_bounds__(GRID_THREADS) grid_kernel(int nA, int64_t gcols, const double* __restrict__ alt,
                                                            const double* __restrict__ grav,
                                                            const double* __restrict__ dalt_c,
                                                            const double* __restrict__ inv_r, double* __restrict__ out) {
  const int64_t col = int64_t(blockIdx.x) * GRID_THREADS + threadIdx.x;
  if (col >= gcols) return;
  const int G = nA + 4, g = blockIdx.y, i = g - 1;
  auto A = [&](int c) { return alt[int64_t(c + 1) * gcols + col]; };
  auto F = [&](int c) { return (c < 0) ? A(0) - A(-1) : A(c) - A(c - 1); };  // dAlt_F(-1) = dAlt_F(0)
  auto R = [&](int c) { return 1.0 / inv_r[int64_t(c + 1) * gcols + col]; };
  auto put = [&](int k, double v) { out[(int64_t(k) * G + g) * gcols + col] = v; };
  const double dF = F(i), idf = 1.0 / dF, dc = dalt_c[int64_t(g) * gcols + col];
  put(GC_DALTF, dF);
  put(GC_H2, idf * 2.0);
  put(GC_IDF, idf);
  put(GC_IDC, 1.0 / dc);
  put(GC_GRAV, grav[int64_t(g) * gcols + col]);
  put(GC_INVR, inv_r[int64_t(g) * gcols + col]);
  put(GC_R, R(i));
  put(GC_ALT, A(i));
  double m[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const bool interior = i >= 1 && i <= nA;
  if (interior) {
    const double h1 = F(i - 1), h2 = F(i), h3 = F(i + 1), h4 = F(i + 2);
    const double H2 = h2 + h1, H3 = h3 + h2 + h1, H4 = h4 + h3 + h2 + h1;
    m[0] = (h2 * h3 * (h3 + h4)) / (h1 * H2 * H3 * H4);
    m[1] = -1.0 * (H2 * h3 * (h3 + h4)) / (h1 * h2 * (h2 + h3) * (h2 + h3 + h4));
    m[3] = H2 * h2 * (h4 + h3) / (H3 * (h2 + h3) * h3 * h4);
    m[4] = -1.0 * H2 * h2 * h3 / (H4 * (h2 + h3 + h4) * (h3 + h4) * h4);
    m[2] = (h2 * h3 * (h3 + h4) + H2 * h3 * (h3 + h4) - H2 * h2 * (h3 + h4) - H2 * h2 * h3) /
           (H2 * h2 * h3 * (h3 + h4));
  }
  for (int k = 0; k < 5; ++k) put(GC_M0 + k, m[k]);
  // boundary meshes: lower cells 0, -1, then upper nAlts+1, nAlts+2
  double* bc = out + int64_t(NGC) * G * gcols + col;
  if (g < 4) {
    const int k = g & 1;
    const bool up = g >= 2;
    const int iAlt = up ? nA + 1 + k : -k;
    const double h1 = up ? F(iAlt - 1) : F(iAlt + 2), h2 = up ? F(iAlt - 2) : F(iAlt + 3);
    const double h3 = up ? F(iAlt - 3) : F(iAlt + 4), h4 = up ? F(iAlt - 4) : F(iAlt + 5);
    const double M1 = h1, M2 = h1 + h2, M3 = h1 + h2 + h3, M4 = h1 + h2 + h3 + h4;
    const double s = up ? 1.0 : -1.0;
    double* o = bc + int64_t(5 * g) * gcols;
    o[0] = s * (M2 * M3 * M4 + M1 * M3 * M4 + M1 * M2 * M4 + M1 * M2 * M3) / (M1 * M2 * M3 * M4);
    o[gcols] = -s * (M2 * M3 * M4) / (h1 * h2 * (h2 + h3) * (h2 + h3 + h4));
    o[2 * gcols] = s * (M1 * M3 * M4) / (M2 * h2 * h3 * (h3 + h4));
    o[3 * gcols] = -s * (M1 * M2 * M4) / (M3 * (h3 + h2) * h3 * h4);
    o[4 * gcols] = s * (M1 * M2 * M3) / (M4 * (h2 + h3 + h4) * (h3 + h4) * h4);
  }
  // AUSM: the Kp / Ku altitude profiles, the spherical face areas and cell
  // volume, the wind-diffusion factor
  double a[NGA] = {dc, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  static_assert(GA_DALTC == 0 && NGA == 7, "the AUSM rows");
  if (interior) {
    const double LeftRadius = 0.5 * (R(i) + R(i - 1));
    const double RightRadius = 0.5 * (R(i) + R(i + 1));
    a[GA_AP] = RightRadius * RightRadius;
    a[GA_AM] = LeftRadius * LeftRadius;
    a[GA_VOL] = (1.0 / 3.0) * (RightRadius * RightRadius * RightRadius - LeftRadius * LeftRadius * LeftRadius);
    const double LogMaxKu = log(0.50), LogMinKu = log(0.25);
    const double LogMaxKp = log(1.0e-09), LogMinKp = log(1.0e-19);
    const double th = tanh((A(i) - 160.0e+03) / 15.0e+03);
    a[GA_KP] = exp(LogMinKp + 0.5 * (LogMaxKp - LogMinKp) * (1.0 + th));
    a[GA_KU] = exp(LogMinKu + 0.5 * (LogMaxKu - LogMinKu) * (1.0 + th));
    a[GA_DAMP] = 0.35 * exp(-1.0 * (A(i) - A(0)) / (45.0e+03));
  }
  double* ga = out + (int64_t(NGC) * G + NBC) * gcols;
  for (int k = 0; k < NGA; ++k) ga[(int64_t(k) * G + g) * gcols + col] = a[k];
}

}  // namespace

cudaError_t grid_launch(int nAlts, int64_t gcols, const double* alt, const double* grav, const double* dalt_c,
                        const double* inv_r, double* out, cudaStream_t stream) {
  if (gcols <= 0) return cudaSuccess;
  const dim3 grid(unsigned((gcols + GRID_THREADS - 1) / GRID_THREADS), unsigned(nAlts + 4));
  void* args[] = {&nAlts, &gcols, &alt, &grav, &dalt_c, &inv_r, &out};
  return cudaLaunchKernel((const void*)grid_kernel, grid, dim3(GRID_THREADS), args, 0, stream);
}

}  // namespace gv
