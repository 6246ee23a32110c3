// hz_kernel.cu -- the horizontal advance (advance_horizontal.f90:58-1034) on
// the GPU: gitm_hz_advance's kernel, in its own translation unit.
//
// One CTA per (block, altitude) plane.  The plane's swept fields (Rho,
// Temperature, Velocity, the six NDensityS and VerticalVelocity, the advected
// IDensityS: 19 fields) and its grid metrics are loaded with their two ghost
// rings from GITM's own Fortran-layout arrays (a plane of one field is
// contiguous there, longitude fastest) into shared memory.  Each of the four
// RK stages of :168-345 is three phases:
//   slopes    the limited slopes of calc_facevalues_lons / _lats (:928-1034),
//             one per field, direction and cell, to shared memory
//   cells     horizontal_solver (:535-818): the face values, the Rusanov
//             gradient and diffusion (calc_rusanov_lons / _lats, :821-922) and
//             the equations, four threads per cell with five fields each
//   update    Orig + c K, each thread its own fields
// The ghost rings keep their values through the stages, as in the reference.
// The store phase writes the interior cells back with the stores of
// :346-421 and, with UseImprovedIonAdvection, the parallel ion-velocity
// divergence of :423-517 (UAM_Gradient, gradient.f90:4-104) at the cell,
// which reads only IVelocityPar and the grid; the CTA of the first and last
// altitude also rewrite the electron sum of the ghost planes.
//
// What bounds it is the FP64 pipe and the latency of its chains.  With one
// thread per cell and every slope formed by each of the three cells that read
// it (486 per field of a 9 x 9 plane instead of 198), 12 warps ran per SM at
// 168 registers, and a 2 degree globe (10,000 planes of 9 x 9) took 3.11 ms;
// with the slopes shared and five fields per thread 1.32 ms.  Both spill: the
// instance of two CTAs of 12 warps, at 80 registers, keeps part of a thread's
// values in local memory.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/gitm_hz.h"
#include "vert_common.cuh"
#include "vert_hz.cuh"
#include "vert_math.cuh"

namespace gv {

namespace {

constexpr int HZ_NSW = 5 + 2 * NS + NADV;  // swept fields
constexpr int NI_ALL = GITM_NIONS - 1;     // ions without the electrons
constexpr int HF_R = 0, HF_T = 1, HF_V = 2, HF_N = 5, HF_W = 5 + NS, HF_I = 5 + 2 * NS;
constexpr int HZ_NGP = 6;   // metric planes with ghost rings: IFB, DFB lon; IFB, DFB lat; cMax E, N
constexpr int HZ_NLD = HZ_NSW + 4;  // planes loaded whole: the fields and the four metrics
constexpr int HZ_PER = 5;   // fields of a thread
constexpr int HZ_GRP = 4;   // threads of a cell: fields 5 g .. 5 g + 4
// A thread takes a line's slopes of up to HZ_LINE cells, HZ_PART of a longer
// one: a line of 128 cells was one thread's chain while the CTA waited (40
// blocks of 128 x 2 cells at 20 altitudes 1,977 us, now 499; 770 with a thread
// per cell).  Parts of 5, 7, 8 and 9 cells, 30 blocks at 10 altitudes: 128 x 2
// 249, 250, 249 and 252 us (343 with a thread per cell), 100 x 2 268, 273, 292
// and 291 (285), 42 x 2 105, 105, 121 and 119 (150): an odd length keeps the
// parts' lanes on different banks.  Ordinary lines stay whole, in instances of
// their own: the parts' index arithmetic cost 9 x 9 blocks 6 %.
constexpr int HZ_LINE = 26;
constexpr int HZ_PART = 5;
constexpr double F1 = 0.6250000;  // Factor1, advance_horizontal.f90:939
constexpr double F2 = 0.0416667;  // Factor2, advance_horizontal.f90:940
static_assert(HZ_PER * HZ_GRP >= HZ_NSW && HF_N == HZ_PER, "the groups' fields");

// Shared-memory plan of one plane (doubles).  Rows of NIp cells and of NLp
// longitude slopes are odd, so lanes on neighbouring rows do not collide
// (padding rows and planes to be free of all collisions gained nothing).  P:
// cells of a plane with ghosts, C: interior cells, per: slopes of a field
// (lines along longitude, then along latitude, longitude fastest).
// batch: the fields whose slopes are held at once, a multiple of HZ_PER (all
// of them for every ordinary block; thin blocks of 2 x 128 cells take fewer).
// keep: Orig and the RK accumulators of the cells are held here too, which
// frees 20 registers of every thread, where there is room.
struct HzLayout {
  int NIp, P, C, NLp, NL, per;
  int S, D, G, K, M, R, stride;  // M: Gamma, RadialDistance, IVelocity east and north of the cells;
                                 // R: sin, cos and tan of the latitude of every interior row
};

__host__ __device__ inline HzLayout hz_layout(int nLons, int nLats, int batch, bool keep) {
  HzLayout L;
  L.NIp = (nLons + 4) | 1;
  L.NLp = (nLons + 2) | 1;
  L.NL = L.NLp * nLats;
  L.P = L.NIp * (nLats + 4);
  L.per = L.NL + (nLats + 2) * nLons;
  L.C = nLons * nLats;
  int o = 0;
  L.S = o;  o += HZ_NSW * L.P;
  L.D = o;  o += (batch < HZ_NSW ? batch : HZ_NSW) * L.per;
  L.G = o;  o += HZ_NGP * L.P;
  L.K = o;  o += keep ? 2 * HZ_NSW * L.C : 0;
  L.M = o;  o += keep ? 4 * L.C : 0;
  L.R = o;  o += 3 * nLats;
  L.stride = o;
  return L;
}

// The limited slopes of cells q0 .. q1 of one line (calc_facevalues_lons /
// _lats; cells 0 .. n+1) of values V and inverse face distances IF, both with
// stride s (index 0 = cell -1), to d with stride sd.  4th-order differences,
// with the 2nd-order one on the outer side of cells 0 and n+1.  Along the line
// each value and each difference is formed once: 3 shared-memory accesses and
// 11 FP64 instructions per slope (9 and 16 with a thread per slope).
__device__ __forceinline__ void hz_slopes(const double* V, const double* IF, double* d, int s, int sd, int q0, int q1,
                                          int n, double beta) {
  double vm = V[q0 * s], v0 = V[(q0 + 1) * s], vp = V[(q0 + 2) * s];  // cells q0-1, q0, q0+1
  // between cells q0-1 and q0; of cell 0 the 2nd-order one
  double dn = IF[(q0 + 1) * s];
  if (q0 == 0)
    dn = (v0 - vm) * dn;
  else
    dn = (dn * 2) * (F1 * (v0 - vm) - F2 * (vp - V[(q0 - 1) * s]));
  const int last = min(q1, n);
#pragma unroll 4
  for (int q = q0; q <= last; ++q) {
    // between cells q and q+1
    const double vq = V[(q + 3) * s];
    const double up = (IF[(q + 2) * s] * 2) * (F1 * (vp - v0) - F2 * (vq - vm));
    d[q * sd] = limiter_mc(up, dn, beta);
    dn = up;
    vm = v0;
    v0 = vp;
    vp = vq;
  }
  if (q1 > n) d[(n + 1) * sd] = limiter_mc((vp - v0) * IF[(n + 3) * s], dn, beta);
}

// A cell's faces along one direction: halves of the face widths, the
// dissipation coefficients times 1 / width, half of 1 / width.
struct HzFaces {
  double h0, h1, b0, b1, g;
  // calc_rusanov_lons / _lats: gradient and diffusion from the slopes of the
  // cell's line neighbours (sm, s0, sp) and their values
  __device__ __forceinline__ void sweep(double vm, double v0, double vp, double sm, double s0, double sp, double& grad,
                                        double& diff) const {
    const double W0 = fma(sm, h0, vm), E0 = fma(-s0, h0, v0);
    const double W1 = fma(s0, h1, v0), E1 = fma(-sp, h1, vp);
    grad = (W1 + E1 - W0 - E0) * g;
    diff = fma(b1, E1 - W1, -(b0 * (E0 - W0)));
  }
  __device__ __forceinline__ double grad(double vm, double v0, double vp, double sm, double s0, double sp) const {
    return (fma(s0, h1, v0) + fma(-sp, h1, vp) - fma(sm, h0, vm) - fma(-s0, h0, v0)) * g;
  }
};

struct HzArgs {
  GitmHzParams prm;
  GitmHzBlocks b;
  double dt;
  uint32_t* status;  // one word per block
  int group;         // threads of a field group: the interior cells rounded up to whole warps
  int batch;         // see hz_layout
  int parts_lon, parts_lat;  // threads that share a line (1, or parts of HZ_PART cells)
  unsigned magic;    // ceil(2^32 / tasks of a field): w / tasks = umulhi(w, magic) for w < 2^16
};

// Threads: HZ_GRP groups of A.group (at most NT in all); thread q of a group
// has interior cell q.  SPLIT: lines of more than HZ_LINE cells are shared by
// threads.
template <int NT, int MINB, bool KEEP, bool SPLIT>
__global__ void __launch_bounds__(NT, MINB) hz_step_kernel(const HzArgs A) {
  extern __shared__ double sm[];
  const GitmHzBlocks& B = A.b;
  const GitmHzParams& prm = A.prm;
  const int nl = B.n_lons, nt = B.n_lats, na = B.n_alts;
  const int NG = nl + 4, NJ = nt + 4, NK = na + 4;
  const int PG = NG * NJ;  // a plane of GITM's arrays
  const int64_t V = int64_t(PG) * NK;
  const int k = blockIdx.x % na + 1;  // Fortran altitude of this plane
  const int b = blockIdx.x / na;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const HzLayout L = hz_layout(nl, nt, A.batch, KEEP);
  const int NI = L.NIp, P = L.P;  // rows and planes in shared memory
  const double dt = A.dt;
  // first element of plane k of field f of a block array with nf fields
  auto plane = [&](const double* a, int f, int nf) -> const double* {
    return a + ((int64_t(b) * nf + f) * NK + (k + 1)) * PG;
  };
  auto lat1 = [&](const double* a, int j) { return a[int64_t(b) * NJ + (j + 1)]; };

  // ---------------------------------------------------------------- load
  double* S = sm + L.S;
  double* D = sm + L.D;
  double* GP = sm + L.G;
  auto src_of = [&](int f) -> const double* {
    if (f == HF_R) return plane(B.rho, 0, 1);
    if (f == HF_T) return plane(B.temperature, 0, 1);
    if (f < HF_N) return plane(B.velocity, f - HF_V, 3);
    if (f < HF_W) return plane(B.ndensity_s, f - HF_N, GITM_NSPECIES_TOTAL);
    if (f < HF_I) return plane(B.vert_vel, f - HF_W, NS);
    if (f < HZ_NSW) return plane(B.idensity_s, f - HF_I, GITM_NIONS);
    return plane(f == HZ_NSW ? B.inv_dlon_dist_fb : f == HZ_NSW + 1 ? B.dlon_dist_fb
                 : f == HZ_NSW + 2 ? B.inv_dlat_dist_fb : B.dlat_dist_fb, 0, 1);
  };
  // a field per warp and turn, straight into shared memory
  for (int f = tid >> 5; f < HZ_NLD; f += nthr >> 5) {
    const double* src = src_of(f);
    double* dst = f < HZ_NSW ? S + f * P : GP + (f - HZ_NSW) * P;
    for (int c = tid & 31; c < PG; c += 32) {
      const int j = c / NG;
      const uint32_t d = uint32_t(__cvta_generic_to_shared(dst + c + j * (NI - NG)));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src + c) : "memory");
    }
  }
  {
    // cMax_GDB(0:nLons+1, 0:nLats+1, 0:nAlts+1, 3, nBlocks): east and north
    // components of this altitude (the outer ghost ring is never read)
    const int ci2 = nl + 2, n = ci2 * (nt + 2);
    for (int w = tid; w < 2 * n; w += nthr) {
      const int d = w >= n, c = w - d * n;
      const int j = c / ci2, i = c - j * ci2;  // Fortran indices
      GP[(4 + d) * P + (j + 1) * NI + i + 1] = B.cmax[((int64_t(b) * 3 + d) * (na + 2) + k) * n + c];
    }
  }
  // what the equations read of other arrays at cell q: Gamma, RadialDistance, IVelocity east, north
  auto other = [&](int m) -> const double* {
    return m == 0 ? plane(B.gamma, 0, 1) : m == 1 ? plane(B.radial_distance, 0, 1) : plane(B.ivelocity, m - 2, 3);
  };
  if (KEEP) {
    for (int w = tid; w < 4 * L.C; w += nthr) {
      const int m = w / L.C, c = w - m * L.C;
      const uint32_t d = uint32_t(__cvta_generic_to_shared(sm + L.M + w));
      const double* src = other(m) + (c / nl + 2) * NG + (c % nl + 2);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    }
  }
  for (int j = tid; j < nt; j += nthr) {
    sm[L.R + 3 * j] = sin(lat1(B.latitude, j + 1));
    sm[L.R + 3 * j + 1] = lat1(B.cos_latitude, j + 1);
    sm[L.R + 3 * j + 2] = lat1(B.tan_latitude, j + 1);
  }
  const int grp = tid / A.group, q = tid - grp * A.group;
  const bool cell = q < L.C;
  const int ci = cell ? q % nl + 1 : 1, cj = cell ? q / nl + 1 : 1;  // Fortran (iLon, iLat)
  const int pc = (cj + 1) * NI + (ci + 1);  // the cell in a plane of shared memory
  const int pg = (cj + 1) * NG + (ci + 1);  // and of GITM's arrays
  // per-cell constants of the equations (:680-686)
  const double* row = sm + L.R + 3 * (cj - 1);
  const double InvR = plane(B.inv_radial_distance, 0, 1)[pg];
  const double beta = prm.beta_limiter;
  const int f0 = grp * HZ_PER;  // this thread's fields
  const int nf = min(HZ_PER, HZ_NSW - f0);
  double orig_r[KEEP ? 1 : HZ_PER], acc_r[KEEP ? 1 : HZ_PER];
  double* keep = sm + L.K + (cell ? f0 * L.C + q : 0);  // Orig of field f0 + j at keep[j C], its accumulator NSW C on
  auto orig = [&](int j) -> double& { return KEEP ? keep[j * L.C] : orig_r[KEEP ? 0 : j]; };
  auto acc = [&](int j) -> double& { return KEEP ? keep[(HZ_NSW + j) * L.C] : acc_r[KEEP ? 0 : j]; };
  HzFaces lo, la;
  {
    const double il = plane(B.inv_dlon_dist_gb, 0, 1)[pg], it = plane(B.inv_dlat_dist_gb, 0, 1)[pg];
    lo.g = 0.5 * il;
    la.g = 0.5 * it;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  {
    const double* DFlo = GP + 1 * P;
    const double* DFla = GP + 3 * P;
    const double* CMe = GP + 4 * P;
    const double* CMn = GP + 5 * P;
    lo.h0 = 0.5 * DFlo[pc];
    lo.h1 = 0.5 * DFlo[pc + 1];
    lo.b0 = fmax(CMe[pc - 1], CMe[pc]) * lo.g;
    lo.b1 = fmax(CMe[pc], CMe[pc + 1]) * lo.g;
    la.h0 = 0.5 * DFla[pc];
    la.h1 = 0.5 * DFla[pc + NI];
    la.b0 = fmax(CMn[pc - NI], CMn[pc]) * la.g;
    la.b1 = fmax(CMn[pc], CMn[pc + NI]) * la.g;
  }
#pragma unroll
  for (int j = 0; j < HZ_PER; ++j)
    if (cell && j < nf) orig(j) = S[(f0 + j) * P + pc];  // Orig (:181-186)

  auto value = [&](int m) { return KEEP ? sm[L.M + m * L.C + q] : other(m)[pg]; };
  // where the cell's slopes stand in a field's slope row
  const int dl = (cj - 1) * L.NLp + ci, dt0 = L.NL + cj * nl + (ci - 1);
  const int per = L.per, lines = SPLIT ? nt * A.parts_lon + nl * A.parts_lat : nl + nt;
  auto sweeps = [&](int f, int fb, double& gLo, double& gLa, double& dd) {
    const double* v = S + f * P + pc;
    const double* d = D + (f - fb) * per;
    double dLo, dLa;
    lo.sweep(v[-1], v[0], v[1], d[dl - 1], d[dl], d[dl + 1], gLo, dLo);
    la.sweep(v[-NI], v[0], v[NI], d[dt0 - nl], d[dt0], d[dt0 + nl], gLa, dLa);
    dd = dLo + dLa;
  };

  // ---------------------------------------------------------------- RK4
#pragma unroll 1
  for (int st = 0; st < 4; ++st) {
    double kv[HZ_PER], DivVel = 0.0;
#pragma unroll
    for (int j = 0; j < HZ_PER; ++j) kv[j] = 0.0;
#pragma unroll 1
    for (int fb = 0; fb < HZ_NSW; fb += A.batch) {
      // slopes, a line of a field per thread, or a part of one where lines are long
      const int n = (min(fb + A.batch, HZ_NSW) - fb) * lines;
      for (int w = tid; w < n; w += nthr) {
        const int f = __umulhi(unsigned(w), A.magic), r = w - f * lines;
        const int lons = SPLIT ? nt * A.parts_lon : nt;
        const bool lat = r >= lons;
        const int len = lat ? nt : nl;
        int x = lat ? r - lons : r;  // row x + 1, or column x + 1
        int q0 = 0, q1 = len + 1;
        if (SPLIT && (lat ? A.parts_lat : A.parts_lon) > 1) {
          const int across = lat ? nl : nt, part = x / across;
          x -= part * across;
          q0 = part * HZ_PART;
          q1 = min(q0 + HZ_PART - 1, q1);
        }
        const int at = lat ? x + 2 : (x + 2) * NI;
        hz_slopes(S + (fb + f) * P + at, GP + (lat ? 2 * P : 0) + at, D + f * per + (lat ? L.NL + x : x * L.NLp),
                  lat ? NI : 1, lat ? nl : 1, q0, q1, len, beta);
      }
      __syncthreads();
      // cells
      if (cell) {
        const double VE = S[(HF_V + 0) * P + pc], VN = S[(HF_V + 1) * P + pc];
        if (fb == 0 && f0 >= HF_N && f0 < HF_W) {
          // DivVel_C (:614-617), for the densities among this thread's fields
          const double* v = S + HF_V * P + pc;
          const double* d = D + HF_V * per;
          DivVel = la.grad(v[P - NI], v[P], v[P + NI], d[per + dt0 - nl], d[per + dt0], d[per + dt0 + nl]) +
                   lo.grad(v[-1], v[0], v[1], d[dl - 1], d[dl], d[dl + 1]) - row[2] * VN * InvR;
        }
        if (f0 < fb || f0 >= fb + A.batch) {
          // another batch's fields
        } else if (grp == 0) {
          const double R = S[HF_R * P + pc], T = S[HF_T * P + pc], VU = S[(HF_V + 2) * P + pc];
          const double TanLat = row[2];
          // each sweep's advection and diffusion as it is formed; pE, pN: the pressure gradients
          double gLo, gLa, dd;
          sweeps(HF_R, fb, gLo, gLa, dd);
          kv[0] = dd - (gLa * VN + gLo * VE);
          const double ToR = T / R;
          double pE = gLo * ToR, pN = gLa * ToR;
          sweeps(HF_T, fb, gLo, gLa, dd);
          kv[1] = dd - (gLa * VN + gLo * VE);
          pE = gLo + pE;
          pN = gLa + pN;
          sweeps(HF_V + 0, fb, gLo, gLa, dd);
          DivVel = gLo;
          kv[2] = dt * (dd - (VN * gLa + VE * gLo + VE * (VU - TanLat * VN) * InvR + pE));
          sweeps(HF_V + 1, fb, gLo, gLa, dd);
          // DivVel_C (:614-617)
          DivVel = gLa + DivVel - TanLat * VN * InvR;
          // :749-759, :765-777, :785-790 and the Coriolis terms of :803-813
          kv[3] = dt * (dd - (VN * gLa + VE * gLo + (VN * VU + TanLat * (VE * VE)) * InvR + pN));
          // :688-694, :817-823
          kv[0] = dt * (kv[0] - R * DivVel);
          kv[1] = dt * (kv[1] - (value(0) - 1) * T * DivVel);
          sweeps(HF_V + 2, fb, gLo, gLa, dd);
          kv[4] = dt * (dd - (VN * gLa + VE * gLo));
          if (prm.use_coriolis) {
            const double SinLat = row[0], CosLat = row[1];
            const double CoriolisSin = SinLat * 2 * prm.omega_body;
            const double CoriolisCos = CosLat * 2 * prm.omega_body;
            const double CentrifugalParameter = (prm.omega_body * prm.omega_body) * CosLat * SinLat;
            kv[2] = kv[2] + dt * (CoriolisSin * VN - CoriolisCos * VU);
            kv[3] = kv[3] - dt * (CentrifugalParameter * value(1) + CoriolisSin * VE);
          }
        } else {
#pragma unroll
          for (int j = 0; j < HZ_PER; ++j) {
            if (j >= nf) continue;
            const int f = f0 + j;
            double gLo, gLa, dd;
            sweeps(f, fb, gLo, gLa, dd);
            // species continuity (:696-703), vertical winds (:794-801), advected ions (:719-736)
            double an = VN, ae = VE;
            if (f >= HF_I) {
              ae = value(2);
              an = value(3);
            }
            double adv = gLa * an + gLo * ae;
            if (f < HF_W) adv = fma(S[f * P + pc], DivVel, adv);
            kv[j] = dt * (dd - adv);
          }
        }
      }
      __syncthreads();  // every read of this batch's slopes, and at last of this stage's state, is done
    }
    // update
    const double ca = (st == 1 || st == 2) ? 2.0 : 1.0, cx = (st < 2) ? 0.5 : 1.0;
    if (cell) {
#pragma unroll
      for (int j = 0; j < HZ_PER; ++j) {
        if (j >= nf) continue;
        const double a = (st == 0) ? kv[j] : acc(j) + ca * kv[j];
        if (st < 3) acc(j) = a;
        const double o = orig(j);
        S[(f0 + j) * P + pc] = (st == 3) ? o + (1.0 / 6.0) * a : cx * kv[j] + o;
      }
    }
    __syncthreads();
  }

  // ---------------------------------------------------------------- store
  auto out = [&](double* a, int f, int n) { return a + ((int64_t(b) * n + f) * NK + (k + 1)) * PG + pg; };
  if (cell) {
    bool neg = false;
#pragma unroll
    for (int j = 0; j < HZ_PER; ++j) {
      if (j >= nf) continue;
      const int f = f0 + j;
      const double v = S[f * P + pc];
      if (f >= HF_I) continue;  // the ions below
      double* o = f == HF_R ? out(B.rho, 0, 1) : f == HF_T ? out(B.temperature, 0, 1)
                : f < HF_N ? out(B.velocity, f - HF_V, 3)
                : f < HF_W ? out(B.ndensity_s, f - HF_N, GITM_NSPECIES_TOTAL) : out(B.vert_vel, f - HF_W, NS);
      if (f == HF_T && B.temp_source)
        B.temp_source[((int64_t(b) * na + (k - 1)) * nt + (cj - 1)) * nl + (ci - 1)] = v - orig(j);
      if (f >= HF_N && f < HF_W) neg = neg || v < 0.0;
      *o = v;
    }
    if (neg) atomicOr(&A.status[b], GITM_ST_NEG_DENSITY);  // the reference stops (:359-372)
    if (prm.use_ion_advection && grp == HZ_GRP - 1) {
      const double CosLat = row[1], TanLat = row[2];
      const bool div = prm.use_improved_ion_advection != 0;
      double change = 0.0;
      if (div) {
        // DivIVelocityLocal at the cell (:423-509): UAM_Gradient's component
        // iDir of IVelocityPar(iDir) plus the latitude and radial terms
        const double* VI = prm.non_magnetic ? B.ivelocity : B.ivelocity_par;
        auto vi = [&](int d, int i, int j, int kk) {
          return VI[((int64_t(b) * 3 + d) * NK + (kk + 1)) * PG + int64_t(j + 1) * NG + (i + 1)];
        };
        double D = 0.0;
        double g = 0.0;
        if (nl > 1) {
          const double InvCosLat = 1. / fmax(CosLat, 0.17);
          const int64_t o = int64_t(b) * nl + (ci - 1);
          g = (B.grad_lon_m[o] * vi(0, ci - 1, cj, k) + B.grad_lon_0[o] * vi(0, ci, cj, k) +
               B.grad_lon_p[o] * vi(0, ci + 1, cj, k)) * InvR * InvCosLat;
        }
        D = D + g;
        g = 0.0;
        if (nt > 1) {
          const int64_t o = int64_t(b) * nt + (cj - 1);
          g = (B.grad_lat_m[o] * vi(1, ci, cj - 1, k) + B.grad_lat_0[o] * vi(1, ci, cj, k) +
               B.grad_lat_p[o] * vi(1, ci, cj + 1, k)) * InvR;
        }
        D = D + g;
        double tl = TanLat;
        if (tl > 5.0) tl = 5.0;
        if (tl < -5.0) tl = -5.0;
        D = D - tl * vi(1, ci, cj, k) * InvR;
        g = 0.0;
        if (na > 1) {
          const double* Rg = B.radial_distance + int64_t(b) * V + pg;
          const double Drp = Rg[int64_t(k + 2) * PG] - Rg[int64_t(k + 1) * PG];
          const double Drm = Rg[int64_t(k + 1) * PG] - Rg[int64_t(k) * PG];
          const double DrmOverDrp = Drm / Drp;
          const double Drr2 = DrmOverDrp * DrmOverDrp;
          const double Bottom = Drm * (1 + DrmOverDrp);
          g = (Drr2 * vi(2, ci, cj, k + 1) - vi(2, ci, cj, k - 1) - (Drr2 - 1) * vi(2, ci, cj, k)) / Bottom;
        }
        D = D + g;
        D = D + 2 * vi(2, ci, cj, k) * InvR;
        D = D * CosLat;
        change = dt * D;
      }
      double e = 0.0;
      for (int s = 0; s < NI_ALL; ++s) {
        double v;
        if (s < NADV) {
          v = S[(HF_I + s) * P + pc];
          if (v < 1.0e2) v = 1.0e2;  // :400-412
          if (div) v = v / (1 + change);
          *out(B.idensity_s, s, GITM_NIONS) = v;
        } else {
          v = *out(B.idensity_s, s, GITM_NIONS);
        }
        e = e + v;
      }
      *out(B.idensity_s, GITM_NIONS - 1, GITM_NIONS) = e;
    }
  }
  // with the divergence term the reference sums the electrons on every cell
  // (:512-515): this plane's ghost ring, and the ghost planes of the block
  if (prm.use_ion_advection && prm.use_improved_ion_advection) {
    auto esum = [&](int64_t off) {  // off: index of a cell in field 0's block array
      double e = 0.0;
      for (int s = 0; s < NI_ALL; ++s) e = e + B.idensity_s[off + int64_t(s) * V];
      B.idensity_s[off + int64_t(GITM_NIONS - 1) * V] = e;
    };
    const int64_t base = int64_t(b) * GITM_NIONS * V;
    for (int c = tid; c < PG; c += nthr) {
      const int i = c % NG - 1, j = c / NG - 1;
      if (i >= 1 && i <= nl && j >= 1 && j <= nt) continue;
      esum(base + int64_t(k + 1) * PG + c);
    }
    if (k == 1)
      for (int64_t c = tid; c < 2 * PG; c += nthr) esum(base + c);  // altitudes -1, 0
    if (k == na)
      for (int64_t c = tid; c < 2 * PG; c += nthr) esum(base + int64_t(na + 2) * PG + c);  // nAlts+1, nAlts+2
  }
}

// exchange_messages_sphere (exchange_messages_sphere.f90:4-95) for one
// (block, altitude) plane: the ghost ring takes the interior cells it
// covers (longitude periodic; across a connected pole the cell mirrored in
// latitude, n_blocks_lon / 2 blocks away -- the neighbours of
// AB_SPH_module.f90:180-370 and the packing of AB_XFER_array_util.f90),
// then the polar ghost rows' horizontal winds and ion velocities change sign
// (:35-76, on every altitude: the CTAs of the first and last altitude also
// take the ghost altitudes), then the checks of :78-88.
__global__ void __launch_bounds__(128) hz_exchange_kernel(const GitmHzExchange X, uint32_t* status) {
  const int nl = X.n_lons, nt = X.n_lats, na = X.n_alts;
  const int NI = nl + 4, NJ = nt + 4, NK = na + 4;
  const int64_t P = int64_t(NI) * NJ;
  const int k = blockIdx.x % na + 1;
  const int b = blockIdx.x / na;
  const int bx = b % X.n_blocks_lon, by = b / X.n_blocks_lon;
  const int64_t NLON = int64_t(nl) * X.n_blocks_lon, NLAT = int64_t(nt) * X.n_blocks_lat;
  const int64_t half = int64_t(X.n_blocks_lon / 2) * nl;
  double* VIw = X.non_magnetic ? X.ivelocity : X.ivelocity_par;
  auto at = [&](double* a, int blk, int f, int nf, int kk, int64_t c) -> double& {
    return a[((int64_t(blk) * nf + f) * NK + (kk + 1)) * P + c];
  };
  for (int c = threadIdx.x; c < P; c += blockDim.x) {
    const int i = c % NI - 1, j = c / NI - 1;  // Fortran (iLon, iLat)
    if (i >= 1 && i <= nl && j >= 1 && j <= nt) continue;
    int64_t G = int64_t(bx) * nl + i, GJ = int64_t(by) * nt + j;  // global 1-based
    if (GJ < 1) {
      if (!X.south_pole) continue;
      GJ = 1 - GJ;
      G += half;
    } else if (GJ > NLAT) {
      if (!X.north_pole) continue;
      GJ = 2 * NLAT + 1 - GJ;
      G += half;
    }
    G = ((G - 1) % NLON + NLON) % NLON + 1;
    const int sbx = int((G - 1) / nl), sby = int((GJ - 1) / nt);
    const int si = int(G - int64_t(sbx) * nl), sj = int(GJ - int64_t(sby) * nt);
    const int sb = sby * X.n_blocks_lon + sbx;
    const int64_t sc = int64_t(sj + 1) * NI + (si + 1);
    // the moved fields in pack_vars_nblk's order (ModSphereInterface.f90:
    // 395-447); every load is issued before the first store (source and
    // destination share arrays, so interleaved pairs would serialise)
    constexpr int NX = 1 + 3 + NS + NS + 3 + GITM_NIONS + 3;
    auto field = [&](int q, int& f, int& nf) -> double* {
      if (q == 0) { f = 0; nf = 1; return X.rho; }
      if (q < 4) { f = q - 1; nf = 3; return X.velocity; }
      if (q < 4 + NS) { f = q - 4; nf = NS; return X.vert_vel; }
      if (q < 4 + 2 * NS) { f = q - 4 - NS; nf = GITM_NSPECIES_TOTAL; return X.ndensity_s; }
      if (q == 4 + 2 * NS) { f = 0; nf = 1; return X.temperature; }
      if (q == 5 + 2 * NS) { f = 0; nf = 1; return X.itemperature; }
      if (q == 6 + 2 * NS) { f = 0; nf = 1; return X.etemperature; }
      if (q < 7 + 2 * NS + GITM_NIONS) { f = q - 7 - 2 * NS; nf = GITM_NIONS; return X.use_ion_advection ? X.idensity_s : nullptr; }
      f = q - 7 - 2 * NS - GITM_NIONS; nf = 3;
      return X.use_ion_advection ? VIw : nullptr;
    };
    double v[NX];
#pragma unroll
    for (int q = 0; q < NX; ++q) {
      int f, nf;
      double* a = field(q, f, nf);
      v[q] = a ? at(a, sb, f, nf, k, sc) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < NX; ++q) {
      int f, nf;
      double* a = field(q, f, nf);
      if (a) at(a, b, f, nf, k, c) = v[q];
    }
  }
  __syncthreads();
  // :35-76 -- Latitude(0) < -pi/2: rows -1:0; Latitude(nLats+1) > pi/2:
  // rows nLats+1:nLats+2; every longitude, every altitude
  const double lat0 = X.latitude[int64_t(b) * NJ + 1];
  const double latn = X.latitude[int64_t(b) * NJ + nt + 2];
  auto flip_plane = [&](int kk, int j0) {
    for (int c = threadIdx.x; c < 2 * NI; c += blockDim.x) {
      const int64_t cc = int64_t(j0 + 1 + c / NI) * NI + c % NI;
      for (int d = 0; d < 2; ++d) {
        at(X.velocity, b, d, 3, kk, cc) = -at(X.velocity, b, d, 3, kk, cc);
        at(VIw, b, d, 3, kk, cc) = -at(VIw, b, d, 3, kk, cc);
      }
    }
  };
  const double PI_ = 3.141592653589793;
  for (int side = 0; side < 2; ++side) {
    const bool polar = side == 0 ? (lat0 < -PI_ / 2.0) : (latn > PI_ / 2.0);
    if (!polar) continue;
    const int j0 = side == 0 ? -1 : nt + 1;
    flip_plane(k, j0);
    if (k == 1) {
      flip_plane(-1, j0);
      flip_plane(0, j0);
    }
    if (k == na) {
      flip_plane(na + 1, j0);
      flip_plane(na + 2, j0);
    }
  }
  // :78-88 on this altitude's interior
  uint32_t w = 0;
  for (int c = threadIdx.x; c < nl * nt; c += blockDim.x) {
    const int64_t cc = int64_t(c / nl + 2) * NI + (c % nl + 2);
    if (at(X.temperature, b, 0, 1, k, cc) < 100.0) w |= GITM_ST_LOW_TEMPERATURE;
    if (at(X.rho, b, 0, 1, k, cc) < 0.0) w |= GITM_ST_NEG_DENSITY;
  }
  if (w) atomicOr(&status[b], w);
}

}  // namespace

cudaError_t hz_exchange_launch(const GitmHzExchange& x, uint32_t* status, cudaStream_t stream) {
  hz_exchange_kernel<<<unsigned(int64_t(x.n_blocks_lon) * x.n_blocks_lat * x.n_alts), 128, 0, stream>>>(x, status);
  return cudaGetLastError();
}

constexpr size_t HZ_MAX_SMEM = 227 * 1024;  // of a CTA on sm_100

static size_t hz_smem(int n_lons, int n_lats, int batch, bool keep) {
  return size_t(hz_layout(n_lons, n_lats, batch, keep).stride) * sizeof(double);
}

// Orig and the accumulators in shared memory, with at least a group's fields
// of slopes, where that fits.
static bool hz_keep(int n_lons, int n_lats) { return hz_smem(n_lons, n_lats, HZ_PER, true) <= HZ_MAX_SMEM; }

// All fields' slopes at once where they fit, else as many as do.
static int hz_batch(int n_lons, int n_lats) {
  const bool keep = hz_keep(n_lons, n_lats);
  int batch = HZ_PER * HZ_GRP;
  while (batch > HZ_PER && hz_smem(n_lons, n_lats, batch, keep) > HZ_MAX_SMEM) batch -= HZ_PER;
  return batch;
}

size_t hz_smem_bytes(int n_lons, int n_lats) {
  return hz_smem(n_lons, n_lats, hz_batch(n_lons, n_lats), hz_keep(n_lons, n_lats));
}

// Threads for the slopes of a line of n cells.
static int hz_parts(int n) { return n + 2 <= HZ_LINE ? 1 : (n + 2 + HZ_PART - 1) / HZ_PART; }

int hz_threads(int n_lons, int n_lats) {
  const int c = n_lons * n_lats;
  return c <= 256 ? HZ_GRP * ((c + 31) / 32 * 32) : 0;
}

template <bool SPLIT>
static const void* hz_kernel(int threads, bool keep) {
  if (!keep) return (const void*)hz_step_kernel<1024, 1, false, SPLIT>;
  return threads <= 384   ? (const void*)hz_step_kernel<384, 2, true, SPLIT>
         : threads <= 768 ? (const void*)hz_step_kernel<768, 1, true, SPLIT>
                          : (const void*)hz_step_kernel<1024, 1, true, SPLIT>;
}

cudaError_t hz_launch(const GitmHzParams& prm, const GitmHzBlocks& b, double dt, uint32_t* status,
                      cudaStream_t stream) {
  HzArgs a;
  a.prm = prm;
  a.b = b;
  a.dt = dt;
  a.status = status;
  const int nt = hz_threads(b.n_lons, b.n_lats);
  a.group = nt / HZ_GRP;
  a.batch = hz_batch(b.n_lons, b.n_lats);
  a.parts_lon = hz_parts(b.n_lons);
  a.parts_lat = hz_parts(b.n_lats);
  const unsigned tasks = unsigned(b.n_lats * a.parts_lon + b.n_lons * a.parts_lat);
  a.magic = unsigned(((uint64_t(1) << 32) + tasks - 1) / tasks);
  const size_t smem = hz_smem_bytes(b.n_lons, b.n_lats);
  // up to 96 cells (9 x 9 blocks, GITM's usual size): two CTAs or more per SM
  const bool keep = hz_keep(b.n_lons, b.n_lats);
  const void* fn = (a.parts_lon > 1 || a.parts_lat > 1) ? hz_kernel<true>(nt, keep) : hz_kernel<false>(nt, keep);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchKernel(fn, dim3(unsigned(int64_t(b.n_blocks) * b.n_alts)), dim3(nt), args, smem, stream);
}

}  // namespace gv
