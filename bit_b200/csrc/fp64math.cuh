// FP64 exponential for the near field's and the direct sums' pair loops, free of branches so that
// the independent pairs of an unrolled loop interleave.
//
// P. T. P. Tang's table-driven method ("Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15(2), 1989).  With L = ln 2 / 64,
// t = n L + r, n = 64 m + j (0 <= j < 64), |r| <= L / 2: exp(t) = 2^m * 2^(j/64) * e^r.  n comes
// from the round-to-integer constant 1.5 * 2^52; r from two FMAs with L split into a double
// and its remainder; e^r - 1 from its Taylor polynomial of degree 5 (truncation below 4e-17
// relative for |r| <= 0.0055); 2^(j/64) from a table of the 64 values as a leading double and
// a trailing correction (computed to 80 digits), combined as lead + (trail + lead (e^r - 1)) as
// Tang does; 2^m is added to the exponent field.  exp_tang is the method for any argument, which
// exp_scaled, the form that the kernels run, is checked beside (mathcheck.cu); domain of exp_tang:
// finite t <= 709, and below t = -707 (exp(t) < 1e-307, where 2^m no longer fits a normal exponent)
// the result is 0.
#pragma once

namespace bit {

// 2^(j/64) for j = 0..63: the double nearest it and the double nearest the remainder
__device__ const double2 kExp2Tab64[64] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.6623882552225p+0, -0x1.bb60987591c34p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55},
};

// 64 / ln 2, and ln 2 / 64 as a double plus the double nearest its remainder
constexpr double kExpInvL = 0x1.71547652b82fep+6;
constexpr double kExpLhi = 0x1.62e42fefa39efp-7;
constexpr double kExpLlo = 0x1.abc9e3b39803fp-62;
constexpr double kRoundShift = 0x1.8p52;  // adding it rounds a double below 2^51 to an integer

// Tang's exp; the table is read through the read-only data cache (a warp's lanes gather
// from 64 entries in eight 128-byte lines).
__device__ __forceinline__ double exp_tang(double t) {
  const double kd = fma(t, kExpInvL, kRoundShift);
  const int n = __double2loint(kd);  // rint(t / L), two's complement in the low word
  const double kf = kd - kRoundShift;
  double r = fma(-kf, kExpLhi, t);
  r = fma(-kf, kExpLlo, r);
  // e^r - 1 = r + r^2/2 + r^3/6 + r^4/24 + r^5/120
  double p = fma(r, 0x1.1111111111111p-7, 0x1.5555555555555p-5);
  p = fma(p, r, 0x1.5555555555555p-3);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  p *= r;
  const double2 s = __ldg(kExp2Tab64 + (n & 63));
  const double v = s.x + fma(s.x, p, s.y);
  const int m = n >> 6;
  const double e = __hiloint2double(__double2hiint(v) + (m << 20), __double2loint(v));
  return n < -65280 ? 0.0 : e;  // m < -1020: exp(t) < 1e-307
}

// The kernels' form: exp(-kappa r), kappa fixed: the argument in units of L = ln 2 / 64
// is r * (64 kappa / ln 2), with that factor as a leading double and a correction, so that
// neither kappa r nor the reduction rounds it: n = rint(r nh), f = r nh - n (one fma, exact)
// + r nl, |f| <= 1/2, and e^(f L) - 1 from the same Taylor polynomial with L^k folded into
// its coefficients.  One operation less than -kappa r and exp_tang, and no rounded product.
// tab: this lane's copy of the table in shared memory (exp_tab_fill): 4 copies of 16-byte
// entries side by side, so that at most two of the 8 lanes served together meet in a bank
// (the gather through L1 took up to eight wavefronts a load; 8 copies were no faster).
// exp(-kappa r) below 1e-307 is 0.  Within 1 ulp of CUDA's exp over 16M arguments on B200.
struct ExpScale {
  double nh, nl;  // -64 kappa / ln 2
};
constexpr double kExpNoUnderflow = 700.0;
constexpr double kExpInvLlo = 0x1.777d0ffda0d24p-50;  // 64 / ln 2 - kExpInvL
__device__ __forceinline__ ExpScale exp_scale(double kappa) {
  ExpScale k;
  k.nh = -kappa * kExpInvL;
  k.nl = fma(-kappa, kExpInvL, -k.nh) - kappa * kExpInvLlo;
  return k;
}
constexpr int kExpTabCopies = 4;
constexpr int kExpTabBytes = 64 * kExpTabCopies * 16;
__device__ __forceinline__ void exp_tab_fill(double2* tab, int tid, int threads) {
  for (int i = tid; i < 64 * kExpTabCopies; i += threads) tab[i] = kExp2Tab64[i / kExpTabCopies];
}
// COPIES: of the table at tab (1: kExp2Tab64 itself).  UF: the result is checked for underflow;
// without, |kappa r| < kExpNoUnderflow is required.
template <bool UF, int COPIES>
__device__ __forceinline__ double exp_scaled(double r, ExpScale k, const double2* tab) {
  const double kd = fma(r, k.nh, kRoundShift);
  const int n = __double2loint(kd);
  const double kf = kd - kRoundShift;
  const double f = fma(r, k.nl, fma(r, k.nh, -kf));
  // (ln 2 / 64)^k / k!, k = 5 .. 1
  double p = fma(f, 0x1.5d87fe78a6731p-40, 0x1.3b2ab6fba4e77p-31);
  p = fma(p, f, 0x1.c6b08d704a0c0p-23);
  p = fma(p, f, 0x1.ebfbdff82c58fp-15);
  p = fma(p, f, 0x1.62e42fefa39efp-7);
  p *= f;
  const double2 s = tab[(n & 63) * COPIES];
  const double v = s.x + fma(s.x, p, s.y);
  const double e = __hiloint2double(__double2hiint(v) + ((n >> 6) << 20), __double2loint(v));
  if (!UF) return e;
  return kd < kRoundShift - 65280.0 ? 0.0 : e;  // below 2^-1020, however far
}

}  // namespace bit
