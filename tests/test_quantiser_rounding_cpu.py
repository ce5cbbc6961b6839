"""The element codes of the quantiser rest on quotients x / denom that are one residual step from the correctly
rounded ones.  That is enough if every bf16 x next to a rounding boundary of e2m1 falls on the same side of it, for
every denominator.  Powers of two change nothing, so all 2^23 significands in [1, 2) are all denominators."""
import os
import subprocess
import tempfile

import numpy as np

SRC = r'''
#include <math.h>
#include <stdio.h>
static int side(float y, float b) { return (y > b) - (y < b); }
int main(void) {
  const float bounds[7] = {.25f, .75f, 1.25f, 1.75f, 2.5f, 3.5f, 5.f};
  const int reps[3] = {-1, 0, 1};
  long bad = 0;
#pragma omp parallel for reduction(+ : bad)
  for (int m = 0; m < (1 << 23) - 1; ++m) {     /* the largest one: see the test */
    const float d = 1.f + (float)m * 0x1p-23f;
    for (int u = 0; u < 3; ++u) {
      float r = 1.f / d;                                   /* rcp.approx.ftz: within one ulp of this */
      if (reps[u]) r = nextafterf(r, reps[u] > 0 ? 2.f : 0.f);
      r = fmaf(fmaf(-d, r, 1.f), r, r);
      for (int k = 0; k < 7; ++k) {
        int e;
        const double t = (double)bounds[k] * d;            /* exact */
        const double s = floor(ldexp(frexp(t, &e), 8));
        for (int j = -1; j <= 2; ++j) {                    /* two bf16 values on either side of the boundary */
          const double n = s + j, n8 = n > 256 ? 2 * n - 256 : n < 128 ? 64 + n / 2 : n;    /* eight bits */
          const float x = (float)ldexp(n8, e - 8), y0 = x * r;
          const float y = fmaf(fmaf(y0, -d, x), r, y0);
          bad += side(y, bounds[k]) != side(x / d, bounds[k]);
        }
      }
    }
  }
  printf("%ld\n", bad);
  return 0;
}'''


def test_one_residual_step_keeps_every_quotient_on_its_side():
    """With any reciprocal that is within one ulp.  Left out: 2 - 2^-23, where a reciprocal one ulp too small puts
    the quotient of .5 on the boundary instead of above it; no bf16 maximum gives that denominator."""
    reachable = {float(np.frexp(np.float32(m / 8) * (np.float32(a) / np.float32(2688)))[0])
                 for a in range(128, 256) for m in range(8, 16)}
    assert 1 - 2 ** -24 not in reachable
    with tempfile.TemporaryDirectory() as d:
        c, exe = os.path.join(d, "t.c"), os.path.join(d, "t")
        open(c, "w").write(SRC)
        subprocess.run(["gcc", "-O2", "-fopenmp", "-mfma", "-ffp-contract=off", c, "-o", exe, "-lm"], check=True)
        assert int(subprocess.run([exe], capture_output=True, text=True, check=True).stdout) == 0


TWO_TERMS = r'''
#include <math.h>
#include <stdio.h>
static int side(float y, float b) { return (y > b) - (y < b); }
static int e4m3(float t) {                     /* round to nearest even, saturating: an index of the value */
  int e;
  if (t > 448.f) t = 448.f;
  if (t < 0x1p-6f) return (int)nearbyintf(t * 512.f);
  const float m = nearbyintf(frexpf(t, &e) * 16.f);
  return (e + 100) * 8 + (int)m;
}
int main(void) {
  const float bounds[7] = {.25f, .75f, 1.25f, 1.75f, 2.5f, 3.5f, 5.f};
  long bad = 0;
  /* elements: x / d from 1 / d in two terms */
#pragma omp parallel for reduction(+ : bad)
  for (int m = 0; m < (1 << 23) - 1; ++m) {     /* the largest one: see the test */
    const float d = 1.f + (float)m * 0x1p-23f;
    for (int u = -1; u < 2; ++u) {
      float r = 1.f / d;                                   /* rcp.approx.ftz: within one ulp of this */
      if (u) r = nextafterf(r, u > 0 ? 2.f : 0.f);
      const float rl = fmaf(-d, r, 1.f) * r;
      for (int k = 0; k < 7; ++k) {
        int e;
        const double t = (double)bounds[k] * d;            /* exact */
        const double s = floor(ldexp(frexp(t, &e), 8));
        for (int j = -1; j <= 2; ++j) {                    /* two bf16 values on either side of the boundary */
          const double n = s + j, n8 = n > 256 ? 2 * n - 256 : n < 128 ? 64 + n / 2 : n;    /* eight bits */
          const float x = (float)ldexp(n8, e - 8);
          bad += side(fmaf(x, r, x * rl), bounds[k]) != side(x / d, bounds[k]);
        }
      }
    }
  }
  /* block scales: every block maximum and tensor maximum, their ratios down to scales that round to zero */
  const float h6 = 1.f / 6.f, l6 = -4.967053731282552e-09f;
  for (int ae = -20; ae <= 20; ae += 8)
    for (int a = 128; a < 256; ++a) {
      const float g = ldexpf(a, ae) / 2688.f, r = 1.f / g, rl = fmaf(-g, r, 1.f) * r;
      for (int be = ae - 22; be <= ae; ++be)
        for (int b = 128; b < 256; ++b) {
          const float x = ldexpf(b, be), t = fmaf(x, h6, x * l6);
          bad += e4m3(fmaf(t, r, t * rl)) != e4m3((x / 6.f) / g);
        }
    }
  printf("%ld\n", bad);
  return 0;
}'''


def test_reciprocals_in_two_terms_keep_every_code_and_block_scale():
    """hi + lo of 1 / denom, 1 / 6 and 1 / g: the same e2m1 codes and e4m3 scales as correctly rounded quotients.  Left
    out as above: the denominator 2 - 2^-23."""
    with tempfile.TemporaryDirectory() as d:
        c, exe = os.path.join(d, "t.c"), os.path.join(d, "t")
        open(c, "w").write(TWO_TERMS)
        subprocess.run(["gcc", "-O2", "-fopenmp", "-mfma", "-ffp-contract=off", c, "-o", exe, "-lm"], check=True)
        assert int(subprocess.run([exe], capture_output=True, text=True, check=True).stdout) == 0


EVERY_SCALE = r'''
#include <math.h>
#include <stdio.h>
#include <string.h>
static int on_boundary(float f) { unsigned u; memcpy(&u, &f, 4); return (u & 0x7ffffu) == 0; }    /* five bits at most */
int main(void) {
  long bad = 0;
#pragma omp parallel for reduction(+ : bad)
  for (int m = 0; m < (1 << 23) - 1; ++m) {     /* the largest one: see the test */
    const float g = 1.f + (float)m * 0x1p-23f, r = 1.f / g, rl = fmaf(-g, r, 1.f) * r;
    for (int b = 128; b < 256; ++b) {
      const float x = (float)b, t = fmaf(x, 1.f / 6.f, x * -4.967053731282552e-09f);
      const float q = x / 6.f / g, y = fmaf(t, r, t * rl);
      bad += q != y && (on_boundary(q) || on_boundary(y));
    }
  }
  printf("%ld\n", bad);
  return 0;
}'''


def test_block_scales_for_every_tensor_scale():
    """A caller's own maximum can give any g = maximum / 2688 but 2 - 2^-23: the quotient of a block maximum is the correctly rounded one, or both
    lie between the same two boundaries of e4m3 (which have five bits)."""
    ones = np.float32(2) - np.float32(2) ** -23
    near = np.float32(float(ones) * 2688)
    assert all(c / np.float32(2688) != ones for c in (np.nextafter(near, np.float32(0)), near, np.nextafter(near, np.float32(1e9))))
    with tempfile.TemporaryDirectory() as d:
        c, exe = os.path.join(d, "t.c"), os.path.join(d, "t")
        open(c, "w").write(EVERY_SCALE)
        subprocess.run(["gcc", "-O2", "-fopenmp", "-mfma", "-ffp-contract=off", c, "-o", exe, "-lm"], check=True)
        assert int(subprocess.run([exe], capture_output=True, text=True, check=True).stdout) == 0
