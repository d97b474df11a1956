// Primordial chemistry network (10 species: H2I, H2II, HI, HII, HM, HeI, HeII, HeIII, de, ge):
// rate interpolation, temperature solve, species sources and the analytic Jacobian, as
// device functions shared by the RHS, Jacobian and fused Newton kernels.
//
// Follows src/raja_primordial_network.cpp (the Dengo "cvklu" network): temperature
// 908-1011, rate interpolation 1044-1248, sources 1305-1375, Jacobian 1518-1867.  The species
// sources are written as reaction fluxes times net stoichiometry, summed in reaction order,
// which is the reference's sum term by term.
#pragma once

#include "common.cuh"
#include "df64.cuh"
#include "weno64.cuh"

namespace gbmv {

constexpr int kNT = 50;      // tables per bin
constexpr int kNRates = 46;  // interpolated per cell (21 rates + 25 cooling terms)
constexpr int kTSize = 1024;

// table rows (order of h5tables.TABLE_NAMES)
enum : int {
  K01, K02, K03, K04, K05, K06, K07, K08, K09, K10, K11, K12, K13, K14, K15, K16, K17, K18, K19,
  K21, K22,
  BREM, CEHEI, CEHEII, CEHI, CIECO, CIHEI, CIHEII, CIHEIS, CIHI, COMPTON, GAEL, GAH2, GAHE, GAHI,
  GAHP, H2LTE, H2MCOOL, H2MHEAT, NCRD1, NCRD2, NCRN, REHEII1, REHEII2, REHEIII, REHII,
  GAMMAH2_1, DGAMMAH2_1, GAMMAH2_2, DGAMMAH2_2
};

struct ChemParams {
  const double* tab;  // device, bin-major: tab[bin * kNT + row]
  // dtab[bin * kNT + row] = tab[(bin + 1) * kNT + row] - tab[bin * kNT + row]: the FP64
  // difference every interpolation in the bin takes, formed once at setup (same rounding)
  const double* dtab;
  // the four H2 adiabatic-index tables for the FP32 temperature iterations, per bin:
  // (float) value and (float)(next - value) of gammaH2_2, dgammaH2_2_dT, gammaH2_1,
  // dgammaH2_1_dT -- the roundings the FP32 iterations apply, done once at setup
  const float* gtab;  // device, gtab[bin * 8 + 2 * table + {0 value, 1 slope}]
  const double2* ltab;  // device, chem_log's table
  double dbin, idbin, lb, tlo, thi, z, zp1_4;
  float dbinf, idbinf, lbf;  // (float) of dbin, idbin, lb
  int nbins;
};

// Natural logarithm of a temperature by table and series (P. T. P. Tang, ACM Trans. Math. Softw. 16
// (1990) 378-400): the entry of the exponent and the seven leading significand bits holds 1/c and
// log(c) near its interval's midpoint c, r = T/c - 1 is below 2^-7.99, and six terms of log(1 + r)
// leave 2^-58.  1/c has 21 bits; its low word holds the high word of what log(c) has beyond a
// double, so that the last addition's rounding is the only other error (0.5 units in the last
// place above T = 2; 1.5 with log(c) a double, one FP64 instruction less).  Nine FP64 instructions
// where the library's logarithm takes ~25.  Temperatures outside [1/4, 2^18) take the library's.
constexpr int kLogLowHi = 0x3FD00000;  // high word of 1/4
constexpr int kLogEntries = 20 * 128;
__device__ __forceinline__ double chem_log(const ChemParams& P, double T) {
  const unsigned q = (unsigned)(__double2hiint(T) - kLogLowHi) >> 13;
  if (q >= (unsigned)kLogEntries) return log(T);
  const double2 e = __ldg(P.ltab + q);
  const double r = fma(T, __hiloint2double(__double2hiint(e.x), 0), -1.0);
  double p = fma(r, -1.0 / 6.0, 1.0 / 5.0);
  p = fma(r, p, -1.0 / 4.0);
  p = fma(r, p, 1.0 / 3.0);
  p = fma(r, p, -0.5);
  return e.y + fma(r * r, p, r + __hiloint2double(__double2loint(e.x), 0));
}

// Table position of a temperature: bin b (clamped to the table) and the interpolation weight
// inside it, log T / dbin = b + w (the tables start at T = 1).  The floor is the product rounded
// down at the unit digit of a large constant, so no conversion instruction (they run at the FP64
// rate) and no division by the bin width is needed.
struct ChemPos {
  int b;
  double w;
};
__device__ __forceinline__ ChemPos chem_pos(const ChemParams& P, double logT) {
  constexpr double kUnit = 6755399441055744.0;  // 1.5 2^52: the last bit is the unit digit
  const double y = __fma_rd(logT, P.idbin, kUnit);
  ChemPos q;
  q.b = __double2loint(y);
  double bd = y - kUnit;
  if ((unsigned)q.b >= (unsigned)P.nbins) {
    q.b = q.b < 0 ? 0 : P.nbins - 1;
    bd = (double)q.b;
  }
  q.w = fma(logT, P.idbin, -bd);
  return q;
}

// One Newton step of the temperature solve ge(T) = ge (src/raja_primordial_network.cpp:908-1011)
// at T: returns dT (the step is T - dT) and the slope of T nsum, so that dge/dT = kb / (rho mh)
// slope.  S: the particles with constant adiabatic index over gamma - 1; gk = ge rho mh / kb.
// The reference's expression divided through by kb / (rho mh): one reciprocal for both adiabatic
// indices and one for the slope where it has seven divisions (~55 FP64 instructions, was 122).
struct ChemTemp {
  double H2_1, H2_2, S, gk, dmh;
};
__device__ __forceinline__ ChemTemp chem_temp_setup(const double (&y)[10]) {
  const double kb = 1.3806504e-16, mh = 1.67e-24, gm1 = 1.0 / (5.e0 / 3.e0 - 1);
  ChemTemp c;
  c.H2_1 = y[0];
  c.H2_2 = y[1];
  const double h = y[2] + y[3] + y[4], he = y[5] + y[6] + y[7];
  c.dmh = fma(2.0, y[0] + y[1], fma(1.00794, h, 4.002602 * he)) * mh;
  c.S = gm1 * (h + he + y[8]);
  c.gk = y[9] * (c.dmh * (1.0 / kb));
  return c;
}
__device__ __forceinline__ double chem_temp_step(const ChemParams& P, const ChemTemp& c, double T,
                                                 double logT, double& slope) {
  const ChemPos q = chem_pos(P, logT);
  const double* lo = P.tab + (long)q.b * kNT;
  const double* dl = P.dtab + (long)q.b * kNT;
  const double x1 = fma(q.w, dl[GAMMAH2_1], lo[GAMMAH2_1]) - 1.0;
  const double x2 = fma(q.w, dl[GAMMAH2_2], lo[GAMMAH2_2]) - 1.0;
  const double dg1 = fma(q.w, dl[DGAMMAH2_1], lo[DGAMMAH2_1]);
  const double dg2 = fma(q.w, dl[DGAMMAH2_2], lo[DGAMMAH2_2]);
  const double r = rcp64_any(x1 * x2);
  const double i1 = r * x2, i2 = r * x1;
  const double a1 = c.H2_1 * i1, a2 = c.H2_2 * i2;
  const double nsum = c.S + (a1 + a2);
  slope = fma(-T, fma(a1 * i1, dg1, (a2 * i2) * dg2), nsum);
  return fma(T, nsum, -c.gk) * rcp64_any(slope);
}
// clamp to the table range; dT/dge from the last slope; log T for the rates: logT + l, the log
// at the last iterate plus that of the last ratio, unless the clamp moved T
__device__ __forceinline__ void chem_temp_finish(const ChemParams& P, const ChemTemp& c,
                                                 double slope, double& Ts, double& logT,
                                                 bool known, double& dTs_ge) {
  const double kb = 1.3806504e-16;
  if (Ts < P.tlo) {
    Ts = P.tlo;
    known = false;
  } else if (Ts > P.thi) {
    Ts = P.thi;
    known = false;
  }
  if (!known) logT = chem_log(P, Ts);
  dTs_ge = c.dmh * rcp64_any(kb * slope);
}

// cvklu_calculate_temperature: ten Newton iterations from the previous T, then clamp.  The
// iterations stop once a step is below 2e-15 T: Newton's error falls by at least 80 per step on
// these tables (interpolated gamma and dgamma/dT are not quite consistent, so the convergence
// ends linear with that factor), so the remaining iterations only move the last bit.  From the
// temperature of a nearby state five iterations reach it where ten ran.
__device__ __forceinline__ void chem_temperature(const ChemParams& P, const double (&y)[10],
                                                 double& Ts, double& dTs_ge, double& logT) {
  const ChemTemp c = chem_temp_setup(y);
  double T = Ts, slope = 0.0;
  bool known = false;
#pragma unroll 1
  for (int it = 0; it < 10; ++it) {
    logT = chem_log(P, T);
    const double dT = chem_temp_step(P, c, T, logT, slope);
    const double T0 = T;
    T -= dT;
    if (fabs(dT) <= 2e-15 * T0) {
      logT = fma(-dT, rcp_seed(T0), logT);  // log(T / T0) = -dT / T0 to 1e-30
      known = true;
      break;
    }
  }
  Ts = T;
  chem_temp_finish(P, c, slope, Ts, logT, known, dTs_ge);
}

// The same Newton solve with up to `nfloat` iterations in FP32 (table lookups on float copies
// of the four adiabatic-index tables, value and slope per bin, rounded once at setup exactly
// as the iterations would round the FP64 entries) and 10 - nfloat in FP64 (the fused Newton
// 8 + 2, which keeps the carried temperature within ~1e-16 of the FP64 form's; the DIRK's F
// evaluations 9 + 1, ~1e-10 near a table bin edge, far inside the integration tolerance,
// where Newton converges only linearly).  The FP32 stage stops early
// once its step is below 1e-5 T: Newton's error after such a step is ~1e-10 T, inside the
// basin where the two FP64 iterations restore full accuracy (quadratic convergence), so the
// result matches chem_temperature's to rounding whenever the reference's ten iterations
// converge.  From the carried temperature of a nearby state (successive stages, Newton
// iterates) one FP32 iteration usually suffices.
__device__ __forceinline__ void chem_temperature_mixed(const ChemParams& P, const double (&y)[10],
                                                       double& Ts, double& dTs_ge, double& logT,
                                                       int nfloat) {
  const float kb = 1.3806504e-16f, mh = 1.67e-24f, gm1 = 1.5f;
  const float H2_1 = (float)y[0], H2_2 = (float)y[1], H_1 = (float)y[2], H_2 = (float)y[3],
              H_m0 = (float)y[4], He_1 = (float)y[5], He_2 = (float)y[6], He_3 = (float)y[7],
              de = (float)y[8], ge = (float)y[9];
  const float density = 2.f * H2_1 + 2.f * H2_2 + 1.00794f * H_1 + 1.00794f * H_2 +
                        1.00794f * H_m0 + 4.002602f * He_1 + 4.002602f * He_2 + 4.002602f * He_3;
  const float kdm = kb / (density * mh);
  const float lb = P.lbf, idbin = P.idbinf, dbin = P.dbinf;
  float T = (float)Ts;
#pragma unroll 1
  for (int it = 0; it < nfloat; ++it) {
    const float logTf = logf(T);
    int b = (int)(idbin * (logTf - lb));
    b = b <= 0 ? 0 : (b >= P.nbins ? P.nbins - 1 : b);
    const float t1 = lb + b * dbin;
    const float Tdef = (logTf - t1) / dbin;
    const float4 ga = __ldg(reinterpret_cast<const float4*>(P.gtab + (long)b * 8));
    const float4 gb = __ldg(reinterpret_cast<const float4*>(P.gtab + (long)b * 8 + 4));
    const float g2 = ga.x + Tdef * ga.y;
    const float dg2 = ga.z + Tdef * ga.w;
    const float g1 = gb.x + Tdef * gb.y;
    const float dg1 = gb.z + Tdef * gb.w;
    const float i1 = 1.f / (g1 - 1.f), i2 = 1.f / (g2 - 1.f);
    const float nsum = H2_1 * i1 + H2_2 * i2 +
                       gm1 * (H_1 + H_2 + H_m0 + He_1 + He_2 + He_3 + de);
    const float dge_dT = kdm * (T * (-H2_1 * i1 * i1 * dg1 - H2_2 * i2 * i2 * dg2) + nsum);
    const float dge = kdm * T * nsum - ge;
    const float dT = dge / dge_dT;
    T = T - dT;
    if (fabsf(dT) <= 1e-5f * T) break;
  }
  // remaining iterations (and dT/dge) in FP64: chem_temperature's step without its early end
  const ChemTemp c = chem_temp_setup(y);
  double Td = (double)T, T0 = Td, slope = 0.0, dT = 0.0;
#pragma unroll 1
  for (int it = nfloat; it < 10; ++it) {
    T0 = Td;
    logT = chem_log(P, T0);
    dT = chem_temp_step(P, c, T0, logT, slope);
    Td = T0 - dT;
  }
  Ts = Td;
  // log(T / T0) by its series: |dT / T0| is ~1e-5 at most after the FP32 stage, and the first
  // term dropped is below 3e-17 up to 1e-4
  const double e = -dT * rcp64_any(T0);
  const bool known = fabs(e) < 1e-4;
  logT = fma(e, fma(e, fma(e, 1.0 / 3.0, -0.5), 1.0), logT);
  chem_temp_finish(P, c, slope, Ts, logT, known, dTs_ge);
}

// Rates at the temperature of log logT; WithSlopes: also dk, the rates' differences over the
// table bin, which times idbin / T are their T-derivatives (the Jacobian applies that factor
// once per entry that is linear in them).
template <bool WithSlopes>
__device__ __forceinline__ void chem_rates(const ChemParams& P, double logT, double (&k)[kNRates],
                                           double (&dk)[kNRates]) {
  const ChemPos q = chem_pos(P, logT);
  const double* lo = P.tab + (long)q.b * kNT;
  const double* dl = P.dtab + (long)q.b * kNT;
#pragma unroll
  for (int r = 0; r < kNRates; ++r) {
    const double a = __ldg(lo + r), d = __ldg(dl + r);
    k[r] = fma(q.w, d, a);
    if (WithSlopes) dk[r] = d;
  }
}

// The reactant products of the 21 reactions; a flux is its rate times one of them.
__device__ __forceinline__ void chem_products(const double (&y)[10], double (&p)[21]) {
  const double H2_1 = y[0], H2_2 = y[1], H_1 = y[2], H_2 = y[3], H_m0 = y[4], He_1 = y[5],
               He_2 = y[6], He_3 = y[7], de = y[8];
  p[0] = H_1 * de;
  p[1] = H_2 * de;
  p[2] = He_1 * de;
  p[3] = He_2 * de;
  p[4] = p[3];
  p[5] = He_3 * de;
  p[6] = p[0];
  p[7] = H_1 * H_m0;
  p[8] = H_1 * H_2;
  p[9] = H2_2 * H_1;
  p[10] = H2_1 * H_2;
  p[11] = H2_1 * de;
  p[12] = H2_1 * H_1;
  p[13] = H_m0 * de;
  p[14] = p[7];
  p[15] = H_2 * H_m0;
  p[16] = p[15];
  p[17] = H2_2 * de;
  p[18] = H2_2 * H_m0;
  p[19] = p[12] * H_1;
  p[20] = H_1 * H_1 * H_1;
}
// rate table row of each reaction
__device__ __forceinline__ void chem_fluxes(const double (&k)[kNRates], const double (&p)[21],
                                            double (&r)[21]) {
  static_assert(K01 == 0 && K19 == 18 && K21 == 19 && K22 == 20, "rates in reaction order");
#pragma unroll
  for (int m = 0; m < 21; ++m) r[m] = k[m] * p[m];
}

// Net species sources from reaction fluxes (net stoichiometry).
__device__ __forceinline__ void chem_species(const double (&r)[21], double (&s)[9]) {
  // sums that several rows share
  const double p = r[0] - r[1], q = r[9] - r[10], t = r[2] - r[3], u = r[4] - r[5],
               v = r[13] + r[14], x = r[11] + r[12], y = r[19] + r[20];
  s[0] = r[7] + q - x + r[18] + y;
  s[1] = r[8] - q + r[16] - r[17] - r[18];
  s[2] = fma(2.0, x - y + r[15] + r[17], v - p - r[6] - r[7] - r[8] - q + r[18]);
  s[3] = p - r[8] + q - r[15] - r[16];
  s[4] = r[6] - r[7] - v - r[15] - r[16] - r[18];
  s[5] = -t;
  s[6] = t - u;
  s[7] = u;
  s[8] = p + t + u - r[6] + r[7] + v + r[16] - r[17];
}

struct ChemAux {
  double mdens, imdens, cie, h2;
};

// Shared by the gas-energy source and its Jacobian row: G and N, the densities-weighted sums of
// the H2 cooling and of the three-body terms, and the two reciprocals behind the reference's
// quotients 1/G, 1/D, 1/N, 1/F (D = h2lte / G + 1, F = ncrn / N + 1):
//   1/D = G / (h2lte + G),  1/F = N / (ncrn + N).
struct GeTerms {
  double G, N, i1, i2, H13, Hf;
};
__device__ __forceinline__ GeTerms ge_terms(const double (&k)[kNRates], const double (&y)[10]) {
  const double H2_1 = y[0], H_1 = y[2], H_2 = y[3], He_1 = y[5], de = y[8];
  GeTerms t;
  t.G = H2_1 * k[GAH2] + H_1 * k[GAHI] + H_2 * k[GAHP] + He_1 * k[GAHE] + de * k[GAEL];
  t.N = H2_1 * k[NCRD2] + H_1 * k[NCRD1];
  t.i1 = rcp64_any(k[H2LTE] + t.G);
  t.i2 = rcp64_any(k[NCRN] + t.N);
  t.H13 = H_1 * H_1 * H_1;
  t.Hf = t.H13 * k[H2MHEAT] - H2_1 * H_1 * k[H2MCOOL];
  return t;
}

// Gas-energy source (cooling/heating), src/raja_primordial_network.cpp:1371-1375, the terms
// proportional to the electron density summed before the common factor.
__device__ __forceinline__ double chem_ge_source(const ChemParams& P, const double (&k)[kNRates],
                                                 const double (&y)[10], double T,
                                                 const ChemAux& A, const GeTerms& t) {
  const double H2_1 = y[0], H_1 = y[2], H_2 = y[3], He_1 = y[5], He_2 = y[6], He_3 = y[7],
               de = y[8];
  const double he2 = k[CEHEII] + k[CIHEII] + k[REHEII1] + k[REHEII2] + de * (k[CEHEI] + k[CIHEIS]);
  const double L = H_1 * (k[CEHI] + k[CIHI]) + H_2 * k[REHII] + He_1 * k[CIHEI] + He_2 * he2 +
                   He_3 * k[REHEIII] + k[BREM] * (H_2 + He_2 + 4.0 * He_3) +
                   k[COMPTON] * P.zp1_4 * (T - (2.73 * P.z + 2.73));
  const double h2 = 2.01588 * k[CIECO] * A.mdens + k[H2LTE] * A.h2 * (t.G * t.i1);
  return 0.5 * (t.N * t.i2) * t.Hf - A.cie * (H2_1 * h2 + de * L);
}

// The ge row of the Jacobian by H2_1, H_1, H_2, He_1, He_2, He_3, de (over rho, without
// 1/mdensity) and by ge (without dT/dge idbin / T).
struct GeRow {
  double d0, d2, d3, d5, d6, d7, d8, d9;
};
__device__ __forceinline__ void ge_row(const ChemParams& P, const double (&k)[kNRates],
                                       const double (&dk)[kNRates], const double (&y)[10],
                                       double T, double h2oda, double md, const GeTerms& t,
                                       GeRow& g) {
  const double H2_1 = y[0], H_1 = y[2], H_2 = y[3], He_1 = y[5], He_2 = y[6], He_3 = y[7],
               de = y[8];
  const double H1sq = H_1 * H_1;
  // With D = h2lte / G + 1 and F = ncrn / N + 1 every quotient of the ge row is in G, N and the
  // two reciprocals: 1/D = G i1, 1/(D G) = i1, 1/F = N i2, 1/(F N) = i2.
  const double iF = t.N * t.i2, i1h = t.i1 * t.i1 * h2oda, i22 = t.i2 * t.i2;
  const double lteh = k[H2LTE] * k[H2LTE] * i1h;  // h2lte^2 h2oda / (D G)^2
  const double hlteh = H2_1 * lteh;
  const double nf = 0.5 * k[NCRN] * i22 * t.Hf;
  const double chi = k[CEHI] + k[CIHI], h2c = k[CEHEII] + k[CIHEII] + k[REHEII1] + k[REHEII2],
               h2d = k[CEHEI] + k[CIHEIS], bd = k[BREM] * de;
  g.d0 = (nf * k[NCRD2] - k[GAH2] * hlteh - 0.5 * H_1 * k[H2MCOOL] * iF -
              2.01588 * k[CIECO] * md - k[H2LTE] * h2oda * (t.G * t.i1));
  g.d2 = (nf * k[NCRD1] - k[GAHI] * hlteh - chi * de +
              0.5 * (3 * H1sq * k[H2MHEAT] - H2_1 * k[H2MCOOL]) * iF);
  g.d3 = (-k[GAHP] * hlteh - bd - de * k[REHII]);
  g.d5 = (-k[GAHE] * hlteh - k[CIHEI] * de);
  g.d6 = (-bd - de * (h2c + h2d * de));
  g.d7 = (-4.0 * bd - de * k[REHEIII]);
  g.d8 = (-k[GAEL] * hlteh - H_1 * chi - H_2 * k[REHII] - He_1 * k[CIHEI] -
              He_2 * (h2c + 2 * h2d * de) - He_3 * k[REHEIII] -
              k[BREM] * (H_2 + He_2 + 4.0 * He_3) -
              k[COMPTON] * P.zp1_4 * (T - (2.73 * P.z + 2.73)));
  const double dG = H2_1 * dk[GAH2] + H_1 * dk[GAHI] + H_2 * dk[GAHP] + He_1 * dk[GAHE] +
                    de * dk[GAEL];
  const double dN = H2_1 * dk[NCRD2] + H_1 * dk[NCRD1];
  // d/dT of -H2 h2oda h2lte / D and of Hf / (2 F)
  const double gg = 0.5 * (k[NCRN] * dN - dk[NCRN] * t.N) * i22 * t.Hf +
                    0.5 * iF * (t.H13 * dk[H2MHEAT] - H2_1 * H_1 * dk[H2MCOOL]) -
                    H2_1 * (k[H2LTE] * (k[H2LTE] * dG - t.G * dk[H2LTE]) * i1h +
                            h2oda * dk[H2LTE] * (t.G * t.i1));
  g.d9 = gg;
}

// The Newton matrix's part of the Jacobian with every column multiplied by its own variable:
// put(row, col, v), v = J(row, col) y_col in physical units, without the ge row's 1/mdensity and
// the ge column's dT/dge idbin / T y_9.  A flux's derivative by a reactant times that reactant is
// the flux times its order, so the species entries are sums of the fluxes r (no products), and
// scaling by the Dengo scale and unscaling cancel in them.
template <class Put>
__device__ __forceinline__ void chem_matrix(const ChemParams& P, const double (&k)[kNRates],
                                            const double (&dk)[kNRates], const double (&y)[10],
                                            const double (&pr)[21], const double (&r)[21],
                                            double T, const ChemAux& A, const GeTerms& t,
                                            Put&& put) {
  const double H2_1 = y[0], H_1 = y[2], H_2 = y[3], He_1 = y[5], He_2 = y[6], He_3 = y[7],
               de = y[8];
  const double h2oda = A.h2, md = A.mdens;
  const double r1516 = r[15] + r[16], r714 = r[7] + r[14], r1314 = r[13] + r[14],
               r01 = r[0] - r[1], r23 = r[2] - r[3], r45 = r[4] - r[5], r918 = r[9] + r[18];
  put(0, 0, r[19] - r[10] - r[11] - r[12]);
  put(0, 1, r918);
  put(0, 2, fma(3.0, r[20], fma(2.0, r[19], r[7] + r[9] - r[12])));
  put(0, 3, -r[10]);
  put(0, 4, r[7] + r[18]);
  put(0, 8, -r[11]);
  put(1, 0, r[10]);
  put(1, 1, -r918 - r[17]);
  put(1, 2, r[8] - r[9]);
  put(1, 3, r[8] + r[10] + r[16]);
  put(1, 4, r[16] - r[18]);
  put(1, 8, -r[17]);
  put(2, 0, fma(2.0, r[11] + r[12] - r[19], r[10]));
  put(2, 1, fma(2.0, r[17], r[18] - r[9]));
  put(2, 2, fma(-6.0, r[20], fma(-4.0, r[19], fma(2.0, r[12], r[14] - r[7] - r[8] - r[9] - r[0] -
                                                               r[6]))));
  put(2, 3, fma(2.0, r[15], r[1] - r[8] + r[10]));
  put(2, 4, fma(2.0, r[15], r1314 - r[7] + r[18]));
  put(2, 8, fma(2.0, r[11] + r[17], r[13] - r01 - r[6]));
  put(3, 0, -r[10]);
  put(3, 1, r[9]);
  put(3, 2, r[0] - r[8] + r[9]);
  put(3, 3, -r[1] - r[8] - r[10] - r1516);
  put(3, 4, -r1516);
  put(3, 8, r01);
  put(4, 1, -r[18]);
  put(4, 2, r[6] - r714);
  put(4, 3, -r1516);
  put(4, 4, -r[7] - r1314 - r1516 - r[18]);
  put(4, 8, r[6] - r[13]);
  put(5, 5, -r[2]);
  put(5, 6, r[3]);
  put(5, 8, -r23);
  put(6, 5, r[2]);
  put(6, 6, -r[3] - r[4]);
  put(6, 7, r[5]);
  put(6, 8, r23 - r45);
  put(7, 6, r[4]);
  put(7, 7, -r[5]);
  put(7, 8, r45);
  put(8, 1, -r[17]);
  put(8, 2, r[0] - r[6] + r714);
  put(8, 3, r[16] - r[1]);
  put(8, 4, r[7] + r1314 + r[16]);
  put(8, 5, r[2]);
  put(8, 6, r[4] - r[3]);
  put(8, 7, -r[5]);
  put(8, 8, r01 + r23 + r45 - r[6] + r[13] - r[17]);
  {  // species rows by ge: sources with rates replaced by their bin differences
    double q[21], s[9];
    chem_fluxes(dk, pr, q);
    chem_species(q, s);
#pragma unroll
    for (int m = 0; m < 9; ++m) put(m, 9, s[m]);
  }
  GeRow g;
  ge_row(P, k, dk, y, T, h2oda, md, t, g);
  put(9, 0, g.d0 * H2_1);
  put(9, 2, g.d2 * H_1);
  put(9, 3, g.d3 * H_2);
  put(9, 5, g.d5 * He_1);
  put(9, 6, g.d6 * He_2);
  put(9, 7, g.d7 * He_3);
  put(9, 8, g.d8 * de);
  put(9, 9, g.d9);
}

// Analytic Jacobian in physical units, before the inv_scale*scale and time-unit factors;
// rates k and bin differences dk (chem_rates) at the cell temperature.  Each of the 64 nonzeros is handed to
// put(row, col, value) once, already multiplied by the factors the reference applies to that
// entry (1/mdensity on the ge row, dT/dge on the ge column); entries never put are zero.
// Tge: dT/dge times idbin / T.
template <class Put>
__device__ __forceinline__ void chem_jacobian(const ChemParams& P, const double (&k)[kNRates],
                                              const double (&dk)[kNRates], const double (&y)[10],
                                              const double (&pr)[21], double T, double Tge,
                                              const ChemAux& A, const GeTerms& t, Put&& put) {
  const double H2_1 = y[0], H2_2 = y[1], H_1 = y[2], H_2 = y[3], H_m0 = y[4], He_1 = y[5],
               He_2 = y[6], He_3 = y[7], de = y[8];
  const double h2oda = A.h2, md = A.mdens, imd = A.imdens;
#define SETJ(row, col, expr) put(row, col, (expr))
  const double H1sq = H_1 * H_1;
  SETJ(0, 0, -k[K11] * H_2 - k[K12] * de - k[K13] * H_1 + k[K21] * H1sq);
  SETJ(0, 1, k[K10] * H_1 + k[K19] * H_m0);
  SETJ(0, 2, k[K08] * H_m0 + k[K10] * H2_2 - k[K13] * H2_1 + 2 * k[K21] * H2_1 * H_1 +
                 3 * k[K22] * H1sq);
  SETJ(0, 3, -k[K11] * H2_1);
  SETJ(0, 4, k[K08] * H_1 + k[K19] * H2_2);
  SETJ(0, 8, -k[K12] * H2_1);
  SETJ(1, 0, k[K11] * H_2);
  SETJ(1, 1, -k[K10] * H_1 - k[K18] * de - k[K19] * H_m0);
  SETJ(1, 2, k[K09] * H_2 - k[K10] * H2_2);
  SETJ(1, 3, k[K09] * H_1 + k[K11] * H2_1 + k[K17] * H_m0);
  SETJ(1, 4, k[K17] * H_2 - k[K19] * H2_2);
  SETJ(1, 8, -k[K18] * H2_2);
  SETJ(2, 0, k[K11] * H_2 + 2 * k[K12] * de + 2 * k[K13] * H_1 - 2 * k[K21] * H1sq);
  SETJ(2, 1, -k[K10] * H_1 + 2 * k[K18] * de + k[K19] * H_m0);
  SETJ(2, 2, -k[K01] * de - k[K07] * de - k[K08] * H_m0 - k[K09] * H_2 - k[K10] * H2_2 +
                 2 * k[K13] * H2_1 + k[K15] * H_m0 - 4 * k[K21] * H2_1 * H_1 - 6 * k[K22] * H1sq);
  SETJ(2, 3, k[K02] * de - k[K09] * H_1 + k[K11] * H2_1 + 2 * k[K16] * H_m0);
  SETJ(2, 4, -k[K08] * H_1 + k[K14] * de + k[K15] * H_1 + 2 * k[K16] * H_2 + k[K19] * H2_2);
  SETJ(2, 8, -k[K01] * H_1 + k[K02] * H_2 - k[K07] * H_1 + 2 * k[K12] * H2_1 + k[K14] * H_m0 +
                 2 * k[K18] * H2_2);
  SETJ(3, 0, -k[K11] * H_2);
  SETJ(3, 1, k[K10] * H_1);
  SETJ(3, 2, k[K01] * de - k[K09] * H_2 + k[K10] * H2_2);
  SETJ(3, 3, -k[K02] * de - k[K09] * H_1 - k[K11] * H2_1 - k[K16] * H_m0 - k[K17] * H_m0);
  SETJ(3, 4, -k[K16] * H_2 - k[K17] * H_2);
  SETJ(3, 8, k[K01] * H_1 - k[K02] * H_2);
  SETJ(4, 1, -k[K19] * H_m0);
  SETJ(4, 2, k[K07] * de - k[K08] * H_m0 - k[K15] * H_m0);
  SETJ(4, 3, -k[K16] * H_m0 - k[K17] * H_m0);
  SETJ(4, 4, -k[K08] * H_1 - k[K14] * de - k[K15] * H_1 - k[K16] * H_2 - k[K17] * H_2 -
                 k[K19] * H2_2);
  SETJ(4, 8, k[K07] * H_1 - k[K14] * H_m0);
  SETJ(5, 5, -k[K03] * de);
  SETJ(5, 6, k[K04] * de);
  SETJ(5, 8, -k[K03] * He_1 + k[K04] * He_2);
  SETJ(6, 5, k[K03] * de);
  SETJ(6, 6, -k[K04] * de - k[K05] * de);
  SETJ(6, 7, k[K06] * de);
  SETJ(6, 8, k[K03] * He_1 - k[K04] * He_2 - k[K05] * He_2 + k[K06] * He_3);
  SETJ(7, 6, k[K05] * de);
  SETJ(7, 7, -k[K06] * de);
  SETJ(7, 8, k[K05] * He_2 - k[K06] * He_3);
  SETJ(8, 1, -k[K18] * de);
  SETJ(8, 2, k[K01] * de - k[K07] * de + k[K08] * H_m0 + k[K15] * H_m0);
  SETJ(8, 3, -k[K02] * de + k[K17] * H_m0);
  SETJ(8, 4, k[K08] * H_1 + k[K14] * de + k[K15] * H_1 + k[K17] * H_2);
  SETJ(8, 5, k[K03] * de);
  SETJ(8, 6, -k[K04] * de + k[K05] * de);
  SETJ(8, 7, -k[K06] * de);
  SETJ(8, 8, k[K01] * H_1 - k[K02] * H_2 + k[K03] * He_1 - k[K04] * He_2 + k[K05] * He_2 -
                 k[K06] * He_3 - k[K07] * H_1 + k[K14] * H_m0 - k[K18] * H2_2);
  {  // species rows by ge: sources with rates replaced by slopes, times dT/dge
    double r[21], s[9];
    chem_fluxes(dk, pr, r);
    chem_species(r, s);
#pragma unroll
    for (int q = 0; q < 9; ++q) put(q, 9, s[q] * Tge);
  }
  GeRow g;
  ge_row(P, k, dk, y, T, h2oda, md, t, g);
  put(9, 0, g.d0 * imd);
  put(9, 2, g.d2 * imd);
  put(9, 3, g.d3 * imd);
  put(9, 5, g.d5 * imd);
  put(9, 6, g.d6 * imd);
  put(9, 7, g.d7 * imd);
  put(9, 8, g.d8 * imd);
  put(9, 9, g.d9 * imd * Tge);
#undef SETJ
}


}  // namespace gbmv
