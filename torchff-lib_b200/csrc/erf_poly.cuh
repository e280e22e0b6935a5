// FP64 Ewald terms by polynomials: erfcx for pairs, erf(sqrt(y)) / sqrt(y) and its first two
// derivatives for excluded pairs.
//
// Pairs: on a bounded range of u = alpha r - the cutoff bounds it - erfcx(u) = exp(u^2) erfc(u) lies
// between 0.15 and 1 and a polynomial in u gives it to FP64 rounding. With X = exp(-(alpha r)^2) and
// t = 2 alpha / sqrt(pi) the screened Coulomb terms are sums of positive parts:
//
//   f = erfc(alpha r) / r  = X erfcx / r
//   g = -(1/r) df/dr       = (f + t X) / r^2
//   h = -(1/r) dg/dr       = (3 g + 2 alpha^2 t X) / r^2
//
// The argument of X is one product of r^2, so its rounding error is what the terms' relative error
// grows from, 6e-16 to 2.7e-15 at u = 3.7 (with erfc(u) and exp(-u^2) of a rounded u: 1.1e-14).
//
// Excluded pairs: H(y) = erf(sqrt(y)) / sqrt(y) = 2/sqrt(pi) sum_n (-y)^n / (n! (2n + 1)) is entire, and
//
//   -erf(alpha r) / r and its g and h  =  -alpha H,  2 alpha^3 H',  -4 alpha^5 H''
//
// have no cancellation at short range, where excluded pairs are. H'' falls off as y^-5/2, below the
// rounding of its first coefficients: beyond y = 6, h is taken from g as above. Relative errors below
// 1.4e-15. (The same functions as differences, 1/r - alpha H for pairs, would leave the rounding of
// 1/r: 1e-9 of erfc(alpha r) / r at u = 3.7.)
//
// Coefficients: Chebyshev interpolation of the functions on the range in 60 digits, turned into
// powers of z in [-1, 1] (z = 2 u / U - 1, 2 y / Y - 1). Largest deviations: 5e-17 of erfcx, 2e-17 of
// H(0), H'(0), H''(0); the powers' magnitudes sum to the function's value at 0, so Horner's rule loses
// nothing. They sit in constant memory and are operands of the multiply-adds.
//
// erfc with its branches was most of the operations of the FP64 real-space kernels: FP64 evaluation of
// 3000 waters with erfc and exp 198 us, with this 141 to 144 us. The tile kernel then keeps the FP64 pipe
// busy for 44 % of its cycles and issues in 65 % of them, at 22 of 32 lanes (their pair counts differ).
#pragma once

#include "tff_common.cuh"

namespace tff {
namespace {

// Ranges: y up to 7 (alpha rc for an Ewald tolerance of 5e-4: y = 6.91), up to 13.5 (tolerances to
// 7e-7); longer ones use the erfc and exp of the CUDA library.
enum ErfRange { kErfLibrary = 0, kErfShort, kErfLong };

inline ErfRange erf_range(double alpha, double rc) {
  const double y = alpha * alpha * rc * rc;
  if (!(alpha >= 0.0)) return kErfLibrary;
  return y <= 7.0 ? kErfShort : y <= 13.5 ? kErfLong : kErfLibrary;
}

__constant__ double kErfCoefShort[3][22] = {
    {0.53016560624310392044, -0.24804575394428205608, 0.15621947939798946765, -0.095398924094740114783,
     0.05303808010474833148, -0.026429087159398432151, 0.011798638684339819292, -0.0047418665074359449631,
     0.0017268694800964174878, -0.00057368713357666081735, 0.00017496698410621341012, -0.000049275307451028798316,
     0.000012881701418084933445, -3.1406806920758110451e-6, 7.1718822350268534191e-7, -1.5405001929768831966e-7,
     3.1193838746063087415e-8, -5.9124776548074973782e-9, 1.0771174361830625391e-9, -2.1534713336385994291e-10,
     3.5110228861385203779e-11, 0.0},
    {-0.070870215412652047365, 0.089268273941708172523, -0.081770506366913189874, 0.060614948691147206361,
     -0.037755838799389732018, 0.020226237744462344287, -0.0094837330114127032854, 0.0039471302412627742365,
     -0.0014751955105831060174, 0.00049990566400787374824, -0.00015486515491647200513, 0.000044165846713111298093,
     -0.00001166562096721051834, 2.8687310931243223276e-6, -6.5986207319258051771e-7, 1.4262159107269541034e-7,
     -2.9035038578675659919e-8, 5.5282418414776478155e-9, -1.0113194742975839053e-9, 2.0312373841671472061e-10,
     -3.3220552807095445289e-11, 0.0},
    {0.0255052211262023651, -0.046726003638236117466, 0.051955670306690979058, -0.043149530056444088391,
     0.028894625349470647889, -0.016257828019607456853, 0.007894260479213111214, -0.0033718754521952794975,
     0.0012854717306483897377, -0.00044247187504550840836, 0.00013880685397093954973, -0.00003999639959360313775,
     0.000010655512080250146198, -2.6394845700617448475e-6, 6.1089876147104443953e-7, -1.3267788176083738134e-7,
     2.7154523668873639184e-8, -5.249084618230094729e-9, 9.5208719322090926688e-10, -1.6611392578758074991e-10,
     3.1710211315644354698e-11, -4.9708668615547400884e-12},
};
__constant__ double kErfCoefLong[3][27] = {
    {0.38480835634348233396, -0.19174358008610243611, 0.14157816652554184286, -0.11296538872513501668,
     0.09037951193185111216, -0.069913536414615380813, 0.051230881010378456791, -0.035174166697644585388,
     0.022515504053720893255, -0.013419434709936884761, 0.0074529471785371074712, -0.0038646563463942189318,
     0.0018757754056044718303, -0.00085455012039228436573, 0.00036643338555356245045, -0.00014830650084539673492,
     0.000056812361300450976996, -0.000020641049257533862934, 7.1167539600876480957e-6, -2.3444231942053569194e-6,
     7.5060713057142020001e-7, -2.2490977126513415157e-7, 5.6709040590550783717e-8, -1.5999365370818999749e-8,
     7.082827689582454237e-9, -1.7639288075360658102e-9, 0.0},
    {-0.02840645630905221232, 0.041949086377939629528, -0.050206839433393792165, 0.053558229292802319985,
     -0.051787804751524603695, 0.045538560902955338991, -0.036476913613680113495, 0.026685041767582396236,
     -0.017892579593991401964, 0.011041403856022523738, -0.0062979586507273598732, 0.0033347085374996563064,
     -0.0016457994040787005258, 0.00076002123071371413875, -0.00032957279692783112925, 0.00013464061218329328822,
     -0.000051978523241963277504, 0.000019017763310212703041, -6.6088535096982924855e-6, 2.1830786410485044238e-6,
     -6.8974342835481443594e-7, 2.1175097216530560554e-7, -6.1047979743680486832e-8, 1.4962386600022856871e-8,
     -4.0621275142981945773e-9, 1.704378866168313152e-9, -4.1078646834750521435e-10},
    {0.0062146794633984579247, -0.014876100572857454249, 0.023803657463469783391, -0.030689069482381097195,
     0.033732267335396944637, -0.032423923212287432212, 0.027673376650817027314, -0.021206020257602704113,
     0.014721871772075855973, -0.0093303091287191473362, 0.0054343400983137163277, -0.0029258655206082674825,
     0.0014637433952637123088, -0.00068355868935647812244, 0.00029920505052737612965, -0.0001232076749137002829,
     0.000047888827723029465081, -0.000017624654648788029589, 6.1561380598387244925e-6, -2.0426076917383742398e-6,
     6.4794374394156010499e-7, -1.9967904662628801177e-7, 5.7746538525176713259e-8, -1.4174383826438730934e-8,
     3.8592606978322097887e-9, -1.627100033618517895e-9, 3.9291631250974622532e-10},
};

// erfcx(u) in powers of 2 u / U - 1, U^2 = 7 and 13.5.
__constant__ double kErfcxCoefShort[25] = {
    0.3531532283889421921, -0.25666903099916359337, 0.16884734543211193357, -0.10245863316159168163,
    0.05809012323674185174, -0.031057956946421562583, 0.015768763668503901146, -0.0076445966529360104245,
    0.0035543230794671415144, -0.0015906618329095274079, 0.00068728136450534367756,
    -0.00028743979770065836015, 0.00011662078099687772321, -0.000045987926838163079709,
    0.000017657237930247742722, -6.6144335323863888947e-6, 2.4176165993335347268e-6,
    -8.5824052991708958034e-7, 3.0039743907920067315e-7, -1.084835386026760684e-7, 3.6247527418719507079e-8,
    -8.4335147430632918725e-9, 2.8038293758428327001e-9, -2.1707353931562656211e-9, 6.659930472064703272e-10};
__constant__ double kErfcxCoefLong[29] = {
    0.27397089384189582418, -0.22366136339521592096, 0.16979466525754414481, -0.12120007080978147654,
    0.082003378130640144243, -0.052915535116002857712, 0.032723823390237260079, -0.019470579180527974838,
    0.011182424821373752461, -0.0062161155878497081127, 0.0033522585481755089156, -0.0017573680810650316636,
    0.00089712702790560685137, -0.00044665777265440253939, 0.00021718571179207336212,
    -0.00010328123783356989007, 0.000048067829252725247285, -0.000021880191198089287871,
    9.789641006485781542e-6, -4.3646411342156628541e-6, 1.8781603296814997535e-6, -7.1973030617069291164e-7,
    3.0365900537636943908e-7, -1.8515428733865061121e-7, 7.2810666586545844097e-8, 2.5495578952404890615e-9,
    -3.339947450605960353e-10, -9.5918066883621116037e-9, 3.5640640174143862978e-9};

template <int RANGE> struct ErfDegree;  // of H, H', H'', of erfcx; ends of the range in y and u
template <> struct ErfDegree<kErfShort> {
  static constexpr int n[3] = {20, 20, 21}, x = 24;
  static constexpr double y = 7.0, u = 2.6457513110645905905;
};
template <> struct ErfDegree<kErfLong> {
  static constexpr int n[3] = {25, 26, 26}, x = 28;
  static constexpr double y = 13.5, u = 3.6742346141747672955;
};

// K-th derivative of H at z = 2 y / Y - 1.
template <int RANGE, int K>
__device__ __forceinline__ double erf_poly(double z) {
  constexpr int n = ErfDegree<RANGE>::n[K];
  const auto c = [](int i) { return RANGE == kErfShort ? kErfCoefShort[K][i] : kErfCoefLong[K][i]; };
  double v = c(n);
#pragma unroll
  for (int i = n - 1; i >= 0; --i) v = fma(v, z, c(i));
  return v;
}

// 1/x from y = 1/sqrt(x): the square of y, corrected once (its rounding errors would be multiplied
// by six in the repulsion).
__device__ __forceinline__ double rcp_newton(double x, double y) {
  const double v = y * y;
  return fma(v, fma(-x, v, 1.0), v);
}

template <int RANGE>
__device__ __forceinline__ double erfcx_poly(double z) {
  constexpr int n = ErfDegree<RANGE>::x;
  static_assert(n % 2 == 0, "the even chain starts at the highest power");
  const auto c = [](int i) { return RANGE == kErfShort ? kErfcxCoefShort[i] : kErfcxCoefLong[i]; };
  // even and odd powers apart: two chains half as long (143.8 -> 141.4 us of that evaluation)
  const double w = z * z;
  double even = c(n), odd = c(n - 1);
#pragma unroll
  for (int i = n - 2; i >= 0; i -= 2) even = fma(even, w, c(i));
#pragma unroll
  for (int i = n - 3; i >= 1; i -= 2) odd = fma(odd, w, c(i));
  return fma(odd, z, even);
}

// Terms f, g, h of one pair (see above); excluded pairs: of -erf(alpha r) / r.
template <int RANGE>
struct EwaldPoly {
  double a, y, u, t, a3;  // alpha, alpha^2, 2 alpha / U, 2 alpha / sqrt(pi), 2 alpha^3
  __device__ __forceinline__ explicit EwaldPoly(double alpha) {
    a = alpha;
    y = alpha * alpha;
    u = alpha * (2.0 / ErfDegree<RANGE>::u);
    t = 2.0 * alpha / 1.7724538509055160273;
    a3 = 2.0 * alpha * y;
  }
  // tx: t X
  __device__ __forceinline__ void eval(double r2, double rinv, double rinv2, double &f, double &g, double &tx) const {
    const double x = exp(-y * r2);
    f = x * erfcx_poly<RANGE>(fma(r2 * rinv, u, -1.0)) * rinv;
    tx = t * x;
    g = (f + tx) * rinv2;
  }
  __device__ __forceinline__ double second(double rinv2, double g, double tx) const {
    return fma(2.0 * y, tx, 3.0 * g) * rinv2;
  }
  __device__ __forceinline__ double z(double r2) const { return fma(r2, y * (2.0 / ErfDegree<RANGE>::y), -1.0); }
  __device__ __forceinline__ void excluded(double r2, double &f, double &g) const {
    f = -a * erf_poly<RANGE, 0>(z(r2));
    g = a3 * erf_poly<RANGE, 1>(z(r2));
  }
  __device__ __forceinline__ double excluded_second(double r2, double g) const {
    if (y * r2 > 6.0) return second(1.0 / r2, g, t * exp(-y * r2));
    return -2.0 * a3 * y * erf_poly<RANGE, 2>(z(r2));
  }
};

}  // namespace
}  // namespace tff
