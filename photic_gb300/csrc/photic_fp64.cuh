// photic_fp64.cuh -- the HOPE forward model and the photic cost in IEEE
// double precision, written in the reference's association order.
//
// This translation unit family is compiled with --fmad=false, so no
// multiply-add pair below is fused: every product and sum is rounded
// separately, as in the reference built for x86-64.  Where fused
// multiply-adds are wanted (the FP32 and double-float paths) they are
// written as explicit fma calls.
//
// The exponentials and the divisions by fixed divisors (pi, 120, the band
// count) come from photic_fastmath.cuh: the divisions give the IEEE
// quotient bit for bit with a third of the FP64-pipe work, the exponential
// is within 1 ulp of the host libm's (the reference's) and equal to it on
// 97 % of arguments, against 94.6 % for CUDA's exp.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "photic_fastmath.cuh"
#include "photic_params.h"
#include "photic_softfp.cuh"

#if defined(__CUDACC__)
#define PHOTIC_NOINLINE __noinline__
#else
#define PHOTIC_NOINLINE inline
#endif

namespace photic {

constexpr double kPi = 3.141592653589793;  // model/common.h:19

// Library functions that run once a pixel or a start, out of line: the
// kernels' loops stay within the instruction cache (32 KB streams at full
// rate, beyond it a warp instruction was measured at two to eight times the
// clocks).
static __device__ PHOTIC_NOINLINE double pow_call(double a, double b) { return pow(a, b); }
static __device__ PHOTIC_NOINLINE double div_call(double a, double b) { return sf::div(a, b); }

// Measured-spectrum constants of one pixel and scene that do not change
// during the fit: the Y exponent depends only on the measured
// Rrs(440)/Rrs(490) (model/samodel.c:2897-2902), so pow(440/lambda, Y) is
// evaluated once per pixel instead of once per band evaluation.
template <int NB>
struct PixelF64 {
  double rrs[NB];
  double pw[NB];  // pow(440/lambda, Y)
  double mean;           // mean measured Rrs over the bands
  double r490, r550, r640;
};

// interp_1d at a pre-resolved segment (model/common.c:332-334).
template <int NB>
__device__ __forceinline__ double interp_plan(const InterpPlan &p, const double (&y)[NB]) {
  double y0 = y[0], y1 = y[0];
#pragma unroll
  for (int b = 0; b < NB; b++) {
    if (b == p.i0) y0 = y[b];
    if (b == p.i1) y1 = y[b];
  }
  if (p.exact) return y0;
  return y0 * p.one_minus_t + y1 * p.t;
}

// Per-pixel set-up: Rrs at 440..640 nm with the negative-440 guard
// (model/samodel.c:1785-1799), Y and the spectral mean; and the bands' powers.
template <int NB>
__device__ __forceinline__ double pixel_shape_f64(const FitParams &fp, const double *r,
                                                  PixelF64<NB> &px) {
  const int nb = fp.n_bands;
  double tot = 0.0;
#pragma unroll
  for (int b = 0; b < NB; b++) {
    px.rrs[b] = 0.0;
    if (b < nb) {
      px.rrs[b] = r[b];
      tot = tot + px.rrs[b];
    }
  }
  double r440 = interp_plan(fp.plan[0], px.rrs);
  px.r490 = interp_plan(fp.plan[1], px.rrs);
  px.r550 = interp_plan(fp.plan[2], px.rrs);
  px.r640 = interp_plan(fp.plan[3], px.rrs);
  if (r440 < 0.0) r440 = 0.0001;
  double chi = r440 / px.r490;
  double Y = 3.44 * (1.0 - 3.17 * fm::exp_t(-2.01 * chi));
  if (Y < 0.0) Y = 0.0;
  if (Y > 2.5) Y = 2.5;
  px.mean = tot / (double)nb;
  return Y;
}
template <int NB>
__device__ __forceinline__ void pixel_setup_f64(const FitParams &fp, const SceneConsts &sc,
                                                const double *r, PixelF64<NB> &px) {
  const double Y = pixel_shape_f64<NB>(fp, r, px);
#pragma unroll 1
  for (int b = 0; b < fp.n_bands; b++) px.pw[b] = pow_call(sc.ratio440[b], Y);
}

// Whether a K takes part in the minimum: the reference compares it, cast to
// float, with zero (model/samodel.c:2698), and a double rounds to float zero
// up to 2^-150.
__device__ __forceinline__ bool k_counts(double K) {
  return (fm::bits(K) & 0x7fffffffffffffffLL) > 0x3690000000000000LL;
}

// Depth-dependent K penalty and very-high-K penalty
// (model/samodel.c:2696-2732) for one scene whose min K is K_min.
__device__ __forceinline__ double k_penalty_f64(const KPenalty &kp, double H, double K_min) {
  double e = 0.0;
  if (sf::lt(H, 5.0)) {  // every band of depth below needs it
    int c = -1;
    if (sf::lt(H, 1.0) && sf::lt(K_min, kp.k_thr[0])) c = 0;
    else if (sf::lt(H, 2.0) && sf::lt(K_min, kp.k_thr[1])) c = 1;
    else if (sf::lt(H, 3.0) && sf::lt(K_min, kp.k_thr[2])) c = 2;
    else if (sf::lt(H, 4.0) && sf::lt(K_min, kp.k_thr[3])) c = 3;
    else if (sf::lt(K_min, kp.k_thr[4])) c = 4;
    if (c >= 0) {
      double d = sf::div(1.0, 0.01 + K_min) - kp.inv_t[c];
      e = e + 100.0 * (d * d);
    }
  }
  return e;
}

// One band term of the cost: samodel_Rrs (model/samodel.c:2846-2949) for one
// band, region and scene, and its squared residual (:2571).
struct BandTerm {
  double K;      // diffuse attenuation, clamped to [0, 2.5]
  double rrs_B;  // bottom part of the subsurface reflectance
  double rrs;    // subsurface reflectance
  double Rm;     // modelled Rrs
  double dd;     // (Rm - measured)^2
};

// With every operation compiled (any operands).
static __device__ PHOTIC_NOINLINE void band_term_general(const SceneConsts &sc, int b, double sec_sun,
                                                      double H, double rho, double P, double lnP,
                                                      double G, double X, double pw, double r,
                                                      BandTerm *t) {
  const double a_phi = (sc.a0[b] + sc.a1[b] * lnP) * P;
  const double a_g = G * sc.eS[b];
  const double a = sc.aw[b] + a_phi + a_g;
  const double bb = sc.bbw[b] + X * pw;
  const double u = bb / (a + bb);
  double K = a + bb;
  if (K < 0.0) K = 0.0;
  if (K > 2.5) K = 2.5;
  const double rrs_dp = (0.084 + 0.170 * u) * u;
  const double DuC = 1.03 * sqrt(1.0 + 2.4 * u);
  const double DuB = 1.04 * sqrt(1.0 + 5.4 * u);
  double M = sec_sun + DuC * sc.sec_view;
  const double rrs_C = rrs_dp * (1.0 - fm::exp_t(-M * K * H));
  M = sec_sun + DuB * sc.sec_view;
  const double rrs_B = fm::div_by(rho, kPi, fm::kInvPi) * fm::exp_t(-M * K * H);
  const double rrs = rrs_C + rrs_B;
  const double Rm = 0.5 * rrs / (1.0 - 1.5 * rrs);
  const double d = Rm - r;
  t->K = K;
  t->rrs_B = rrs_B;
  t->rrs = rrs;
  t->Rm = Rm;
  t->dd = d * d;
}

// The same bits with the divisions, square roots, comparisons and most of the
// exponentials on the integer and FP32 pipes (photic_softfp.cuh).  The
// products stay on the FP64 pipe: thirty integer instructions each beside it
// cost more in instruction fetch than they saved (1024 x 320 scene 346 -> 316
// ms without them, 41 x 29 general fit 335 -> 294, 8 009 stacks 217 -> 201).
// A product by the unit secant of a nadir view is skipped (exact).
// The soft operations need normal operands of moderate exponent: the tests
// below cover each, and a term that fails one (an exact zero, an absurd
// exponent, NaN) is evaluated again above.

// The band's medium: u and K, and whether its operands are moderate.
__device__ __forceinline__ bool band_medium(const SceneConsts &sc, int b, double P, double lnP,
                                            double G, double X, double pw, double &u, double &K) {
  const double a_phi = (sc.a0[b] + sc.a1[b] * lnP) * P;
  const double a_g = G * sc.eS[b];
  const double a = sc.aw[b] + a_phi + a_g;
  const double bb = sc.bbw[b] + X * pw;
  const double ab = a + bb;
  u = sf::div_mid(bb, ab);
  K = fm::bits(ab) > 0x4004000000000000LL ? 2.5 : ab;  // > 2.5 (positive here)
  return sf::near_positive(bb) && sf::near_positive(ab) && sf::near_positive(u);
}

// exp(-d) of a light path of d optical depths.  Beyond 200 of them the
// exponentials change no bit of band_close's sums (the columns' part is 1 - 0,
// the bottom's share is lost in rrs): -200 stands for every such depth,
// unless the bottom's part itself is asked for.  (One lane in eight warps was
// that deep, and took its warp through the general term.)
__device__ __forceinline__ double path_loss(double d, bool &deep, bool &ok) {
  deep = fm::bits(d) > 0x4069000000000000LL;
  ok = ok && sf::near_positive(d);
  return sf::exp_neg(deep ? -200.0 : -d, ok);
}

// The term from the two paths' losses; false if it has to be evaluated again.
__device__ __forceinline__ bool band_close(double u, double K, double eC, double eB, bool deepB,
                                           double rho, double r, BandTerm &t) {
  const double rrs_dp = (0.084 + 0.170 * u) * u;
  const double rrs_C = rrs_dp * (1.0 - eC);
  const double rho_pi = fma(rho, fm::kPiHi, rho * fm::kPiLo);
  const double rrs_B = rho_pi * eB;
  const double rrs = rrs_C + rrs_B;
  const double den = 1.0 - 1.5 * rrs;
  const double Rm = sf::div_mid(sf::half_mid(rrs), den);
  const double d = Rm - r;
  t.K = K;
  t.rrs_B = rrs_B;
  t.rrs = rrs;
  t.Rm = Rm;
  t.dd = d * d;
  bool ok = sf::near_positive(rho) && sf::near_positive(rrs) && sf::near(den);
  // (deep: rrs_B at most 2^90 2^-288, below half an ulp of rrs above 2^-90)
  if (deepB) ok = ok && sf::lt(rho_pi, 0x1p90) && sf::lt(0x1p-90, rrs);
  return ok;
}

// A spectrum with a NaN has a NaN mean, and the cost divides by the mean: it is
// NaN whatever the bands' terms.
__device__ __forceinline__ bool nan_mean(double mean) {
  return (fm::bits(mean) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}

// A term that band_close could not give: with every operation, or, for a cost
// that is NaN anyhow, as NaN.  (Pixels with a NaN run every start to its limit
// and fail at every term.  256 pixels in sequence with such a one: 536 ms with
// every operation compiled, 644 with both terms, 293 without the second.)
__device__ __forceinline__ void band_term_again(const SceneConsts &sc, int b, double sec_sun,
                                                bool want, double mean, double H, double rho,
                                                double P, double lnP, double G, double X,
                                                double pw, double r, BandTerm &t) {
  if (!want && nan_mean(mean)) {
    t.dd = mean;
    return;
  }
  BandTerm g;
  band_term_general(sc, b, sec_sun, H, rho, P, lnP, G, X, pw, r, &g);
  t = g;
}

// `want`: more than t.dd and t.K is used.  mean: the spectra's, which the cost
// divides by.
__device__ __forceinline__ void band_term(const SceneConsts &sc, int b, double sec_sun, bool want,
                                          double mean, double H, double rho, double P, double lnP,
                                          double G, double X, double pw, double r, BandTerm &t) {
  double u, K;
  bool ok = band_medium(sc, b, P, lnP, G, X, pw, u, K);
  double DuC = 1.03 * sf::sqrt_mid(1.0 + 2.4 * u);
  double DuB = 1.04 * sf::sqrt_mid(1.0 + 5.4 * u);
  if (sc.sec_view != 1.0) {
    DuC = DuC * sc.sec_view;
    DuB = DuB * sc.sec_view;
  }
  bool deepC, deepB;
  const double eC = path_loss((sec_sun + DuC) * K * H, deepC, ok);
  const double eB = path_loss((sec_sun + DuB) * K * H, deepB, ok);
  ok = band_close(u, K, eC, eB, deepB, rho, r, t) && ok && !(deepB && want);
  if (!ok) band_term_again(sc, b, sec_sun, want, mean, H, rho, P, lnP, G, X, pw, r, t);
}

struct CostDetailsF64 {
  double rrs_error, model_error, bottom_albedo, K_min, iod;
  double Rm[kMaxBands];
};

// What a plain evaluation can keep, besides its cost, so that the products
// at the kept optimum (model/samodel.c:2413, 1994-2079) follow from the same
// evaluation: the Rrs error, K minimum and albedo and, on the lanes that ask
// (want), the index of optical depth's sum and the modelled Rrs.  NoKeep
// keeps nothing.
struct NoKeep {};
template <int NB>
struct BandKeep {
  bool want;
  double iod, Rm[NB];
  double E, K_min, qB;
};

// The cost of one scene and region from its squared residuals' sum and least
// K (model/samodel.c:2696-2744).
__device__ __forceinline__ double cost_total_f64(const FitParams &fp, double err, double K_min,
                                                 double mean, double H, double &E) {
  const int nb = fp.n_bands;
  const double ms = (nb & (nb - 1)) == 0 ? fm::div_count(err, nb)
                                         : fm::div_const(err, (double)nb, fp.inv_nb, fp.inv_nb_lo);
  E = sf::div(100.0 * sf::sqrt(ms), mean);
  double Ke = k_penalty_f64(fp.kp, H, K_min);
  if (sf::lt(0.7, K_min)) {
    double d = 4.0 * (K_min - 0.7);
    Ke = Ke + 100.0 * (d * d);
  }
  const double model = 80.0 * E + 15.0 * Ke;
  return fm::div_120(model);
}

// Cost of x = (H, 100B, q, 100P, 100G, 100X) for one scene, one region,
// one bottom type: samodel_error (model/samodel.c:2432-2759) over
// samodel_Rrs (model/samodel.c:2846-2949).  With one region the depth and
// bottom continuity terms are identically zero and SAM is compiled out.
template <bool kDetails, int NB, class Keep = NoKeep>
__device__ __forceinline__ double cost_f64(const FitParams &fp, const SceneConsts &sc,
                                           const PixelF64<NB> &px, const double *x,
                                           CostDetailsF64 *det, Keep *keep = nullptr) {
  constexpr bool kKeep = !std::is_same<Keep, NoKeep>::value;
  const int nb = fp.n_bands;
  const double H = fabs(x[0]);
  const double B = 0.01 * fabs(x[1]);
  const double qa = fabs(x[2]);
  const double q = fm::self_ratio(qa);  // q / sum(q) with one bottom type
  const double P = 0.01 * fabs(x[3]);
  const double G = 0.01 * fabs(x[4]);
  const double X = 0.01 * fabs(x[5]);
  const double lnP = log(P);
  const double qB = q * B;
  double err = 0.0, K_min = 1.0e4, iod = 0.0;
#pragma unroll 1
  for (int b = 0; b < nb; b++) {
    BandTerm t;
    bool want_B = kDetails;
    if constexpr (kKeep) want_B = keep->want;
    band_term(sc, b, sc.sec_sun, want_B, px.mean, H, qB * sc.refl[b], P, lnP, G, X, px.pw[b],
              px.rrs[b], t);
    err = err + t.dd;
    if (k_counts(t.K) && sf::lt(t.K, K_min)) K_min = t.K;
    if (kDetails) {
      iod = iod + sf::div(t.rrs_B, t.rrs);
      det->Rm[b] = t.Rm;
    }
    if constexpr (kKeep) {
      if (keep->want) {
        iod = iod + sf::div(t.rrs_B, t.rrs);
        keep->Rm[b] = t.Rm;
      }
    }
  }
  double E;
  const double model = cost_total_f64(fp, err, K_min, px.mean, H, E);
  if constexpr (kKeep) {
    keep->E = E;
    keep->K_min = K_min;
    keep->qB = qB;
    keep->iod = iod;
  }
  if (kDetails) {
    det->rrs_error = E;
    det->model_error = model;
    det->bottom_albedo = qB;
    det->K_min = K_min == 1.0e4 ? 0.0 : K_min;
    det->iod = 100.0 * iod / (double)nb;
  }
  return model;
}

// The cold start of samodel_optimise_one_bottom_combination
// (model/samodel.c:2249-2353) for one region, one scene, one bottom type;
// the depth slot is filled per start.
__device__ __forceinline__ double cold_P(double r490, double r550) {
  return 100.0 * 0.072 * pow_call(r490 / r550, -1.7);
}

template <int NB>
__device__ __forceinline__ void cold_start_f64(const FitParams &fp, const PixelF64<NB> &px,
                                               double *start, double *step) {
  start[1] = 100.0 * 4.0 * px.r490;
  step[1] = 1.5 * start[1];
  start[2] = 1.0;
  step[2] = 0.5 * start[2];
  start[3] = cold_P(px.r490, px.r550);
  start[4] = 1.5 * start[3];
  start[5] = 100.0 * 30.0 * fp.aw640 * px.r640;
  step[3] = 2.0 * start[3];
  step[4] = 2.0 * start[4];
  step[5] = 2.0 * start[5];
}

// samodel_Rrs (model/samodel.c:2846-2949) as the reference calls it: the
// physical parameters as given (fabs only where the reference takes it),
// Y from the caller's Rrs(440)/Rrs(490).  Returns Rrs; writes K.
__device__ __forceinline__ double forward_band_rho_f64(const SceneConsts &sc, int b, double P,
                                                       double G, double X, double rho, double H,
                                                       double Delta, double pw, double *K_out,
                                                       double *parts = nullptr) {
  const double a_phi = (sc.a0[b] + sc.a1[b] * log(fabs(P))) * fabs(P);
  const double a_g = fabs(G) * sc.eS[b];
  const double a = sc.aw[b] + a_phi + a_g;
  const double bb = sc.bbw[b] + X * pw;
  const double u = bb / (a + bb);
  double K = a + bb;
  if (K < 0.0) K = 0.0;
  if (K > 2.5) K = 2.5;
  *K_out = K;
  const double rrs_dp = (0.084 + 0.170 * u) * u;
  const double DuC = 1.03 * sqrt(1.0 + 2.4 * u);
  const double DuB = 1.04 * sqrt(1.0 + 5.4 * u);
  double M = sc.sec_sun + DuC * sc.sec_view;
  const double rrs_C = rrs_dp * (1.0 - fm::exp_t(-M * K * H));
  M = sc.sec_sun + DuB * sc.sec_view;
  const double rrs_B = fm::div_by(rho, kPi, fm::kInvPi) * fm::exp_t(-M * K * H);
  const double rrs = rrs_C + rrs_B;
  if (parts) {  // the intermediates samodel_Rrs stores in model_data
    parts[0] = rho;
    parts[1] = rrs_dp;
    parts[2] = rrs_B;
    parts[3] = rrs;
  }
  return 0.5 * rrs / (1.0 - 1.5 * rrs) + Delta;
}

// The same with one bottom type: rho = (q B) rho_sand(lambda).
__device__ __forceinline__ double forward_band_f64(const SceneConsts &sc, int b, double P,
                                                   double G, double X, double qB, double H,
                                                   double Delta, double pw, double *K_out,
                                                   double *parts = nullptr) {
  return forward_band_rho_f64(sc, b, P, G, X, qB * sc.refl[b], H, Delta, pw, K_out, parts);
}

// (long)(10 * y) of the local-minimum test (model/asa047.c:438-470).  C
// leaves the conversion of NaN or |v| >= 2^63 undefined; the x86-64
// instruction returns LONG_MIN there, and that result is used here so the
// outcome does not depend on the host the reference ran on.
__device__ __forceinline__ long long trunc10(double y) {
  double v = 10.0 * y;
  if (!(v > -9.2233720368547758e18 && v < 9.2233720368547758e18)) return (long long)(-9223372036854775807LL - 1);
  return (long long)v;
}

}  // namespace photic
