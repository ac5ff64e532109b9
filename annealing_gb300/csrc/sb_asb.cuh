// The aSB local sub-steps (UpdateTwice, SB/CUDA_GPU/m2_opt.cu:66-71). The reference evaluates them in
// double, because its constants are double literals, and rounds each assignment to float:
//     x = (float)(x + (detune y) dt);  y = (float)(y - dt (((kerr x) x) x + (detune - amp) x)).
// FP64 is scarce on this part (1.6 FMA per clock and SM, 69 clocks from one to the next, against 119
// and 4 in FP32), and one sub-step is nine dependent operations. So each assignment is first formed as
// an unevaluated FP32 sum hi + lo (error-free products and sums: Dekker, "A floating-point technique for
// extending the available precision", 1971; Knuth's two-sum) whose distance from the double result
// is below `slack`; where every value within slack of hi + lo rounds to hi, hi is the float the double
// evaluation gives. Elsewhere (about 1 in 10^5, and wherever something overflows, is NaN or nears the
// subnormals) the double evaluation itself decides, so the bits are always its.
//   * Rounding: the double path makes at most six roundings of 2^-53 relative to the terms' magnitudes,
//     the FP32 one at most eight of 2^-47; slack is 2^-42 of the magnitudes.
//   * Underflow: a product's error term is lost below 2^-149, at most ten of them an assignment, each then
//     multiplied by dt, by kerr dt or by neither (and by an x below 1: x^2 loses bits only there); the added
//     2^-140 (1 + |dt| + |kerr dt|) covers them. (2^-140 alone does not at kerr = 2^33 or dt = 2^20.)
// Compiles as host code too, for the test that compares both evaluations.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define SB_HD __host__ __device__ __forceinline__
#else
#define SB_HD inline
#endif

namespace sbasb {

#ifdef __CUDA_ARCH__
SB_HD float add(float a, float b) { return __fadd_rn(a, b); }
SB_HD float mul(float a, float b) { return __fmul_rn(a, b); }
SB_HD float fma32(float a, float b, float c) { return __fmaf_rn(a, b, c); }
SB_HD double dadd(double a, double b) { return __dadd_rn(a, b); }
SB_HD double dmul(double a, double b) { return __dmul_rn(a, b); }
#else  // compiled without contraction
SB_HD float add(float a, float b) { return a + b; }
SB_HD float mul(float a, float b) { return a * b; }
SB_HD float fma32(float a, float b, float c) { return fmaf(a, b, c); }
SB_HD double dadd(double a, double b) { return a + b; }
SB_HD double dmul(double a, double b) { return a * b; }
#endif

// a + b = s + e exactly
SB_HD void two_sum(float a, float b, float &s, float &e) {
  s = add(a, b);
  const float bb = add(s, -a);
  e = add(add(a, -add(s, -bb)), add(b, -bb));
}
// a * b = p + e exactly (no underflow)
SB_HD void two_prod(float a, float b, float &p, float &e) {
  p = mul(a, b);
  e = fma32(a, b, -p);
}
// hi + lo, and whether everything within slack of it rounds to hi; lost: the bound on what underflow took
SB_HD bool settled(float sum, float err, float magnitude, float lost, float &hi) {
  float lo;
  two_sum(sum, err, hi, lo);
  const float slack = fma32(magnitude, 0x1p-42f, lost);
  return add(hi, add(lo, slack)) == hi && add(hi, add(lo, -slack)) == hi;
}

SB_HD float x_double(float x, float y, float mts_dt, float detune) {
  return (float)dadd((double)x, dmul(dmul((double)detune, (double)y), (double)mts_dt));
}
SB_HD float y_double(float x, float y, float amp, float mts_dt, float detune, float kerr) {
  const double lx = x;
  const double x3 = dmul(dmul(dmul((double)kerr, lx), lx), lx);
  const double lin = dmul(dadd((double)detune, -(double)amp), lx);
  return (float)dadd((double)y, -dmul((double)mts_dt, dadd(x3, lin)));
}

// Keeps the rarely taken double evaluation behind a branch: without it the compiler evaluates both
// sides and selects, which costs what the FP32 form saves.
#ifdef __CUDA_ARCH__
#define SB_ASB_COLD() asm volatile("")
#else
#define SB_ASB_COLD() ((void)0)
#endif

// The bound above on what underflow takes from an assignment.
SB_HD float underflow_bound(float mts_dt, float kerr) {
  return fma32(add(fabsf(mts_dt), fabsf(mul(kerr, mts_dt))), 0x1p-140f, 0x1p-140f);
}

// lost: underflow_bound of the same constants. A kernel that runs many steps makes it once: formed here, in the chain
// between one step's exchange and the next, it cost a one-launch solve 3 % (n = 2000, 2.51 us a step against 2.43).
SB_HD void local(float &x, float &y, float amp, int m, float mts_dt, float detune, float kerr, float lost) {
  // 0 stays 0 (a spin without a start value, padding): settled() would leave it to the double path
  if (x == 0.0f && y == 0.0f && !signbit(x) && !signbit(y) && isfinite(amp) && isfinite(mts_dt) && isfinite(detune) &&
      isfinite(kerr) && mts_dt >= 0.0f && detune >= 0.0f)
    return;
  float ch, cl;  // detune - amp
  two_sum(detune, -amp, ch, cl);
  for (int s = 0; s < m; ++s) {
    {
      float ph, pl, th, tl, sh, se, hi;
      two_prod(detune, y, ph, pl);
      two_prod(ph, mts_dt, th, tl);
      tl = fma32(pl, mts_dt, tl);
      two_sum(x, th, sh, se);
      if (!settled(sh, add(se, tl), add(fabsf(x), fabsf(th)), lost, hi)) {
        SB_ASB_COLD();
        hi = x_double(x, y, mts_dt, detune);
      }
      x = hi;
    }
    {
      float qh, ql, rh, rl, kh, kl, lh, ll, sh, se, uh, ul, wh, we, hi;
      two_prod(x, x, qh, ql);
      two_prod(qh, x, rh, rl);
      rl = fma32(ql, x, rl);
      two_prod(rh, kerr, kh, kl);
      kl = fma32(rl, kerr, kl);
      two_prod(ch, x, lh, ll);
      ll = fma32(cl, x, ll);
      two_sum(kh, lh, sh, se);
      se = add(se, add(kl, ll));
      two_prod(sh, mts_dt, uh, ul);
      ul = fma32(se, mts_dt, ul);
      two_sum(y, -uh, wh, we);
      const float mag = fma32(fabsf(mts_dt), add(fabsf(kh), fabsf(lh)), fabsf(y));
      if (!settled(wh, add(we, -ul), mag, lost, hi)) {
        SB_ASB_COLD();
        hi = y_double(x, y, amp, mts_dt, detune, kerr);
      }
      y = hi;
    }
  }
}
SB_HD void local(float &x, float &y, float amp, int m, float mts_dt, float detune, float kerr) {
  local(x, y, amp, m, mts_dt, detune, kerr, underflow_bound(mts_dt, kerr));
}

}  // namespace sbasb
