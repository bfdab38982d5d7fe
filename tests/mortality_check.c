/*
 * mortality_check.c - checks the binary32 evaluation of the larvae's hourly
 * mortality (sampo_math_fast.h) and the kill thresholds (sampo_model.cuh's
 * formula, given here as the test `(float)v * 2^-32 <= hmr`) against the
 * binary64 definitions of sampo_math.h.
 *
 *   mortality_check STRIDE
 *
 * exp: every STRIDE-th float x in [2^-40, 2.2) and 0; pow: every STRIDE-th
 * float in [0.15, 1); hmr: the whole mortality for x over [0, 4) and some
 * special values. Prints the largest relative error of the unrounded pairs,
 * the binary64 fallbacks and the results that differ (must be 0).
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "sampo_math_fast.h"

static float hmr_definition(float x) {
  float dmr = 0.1f * sampo_expf(x);
  dmr = sampo_fminf(dmr, 0.8f);
  const float dsr = 1.0f - dmr;
  return 1.0f - sampo_powf(dsr, 1.0f / 24.0f);
}

int main(int argc, char** argv) {
  const uint32_t stride = argc > 1 ? (uint32_t)strtoul(argv[1], NULL, 10) : 1u;
  double ee = 0, pe = 0;
  long long ef = 0, em = 0, pf = 0, pm = 0, hm = 0, en = 0, pn = 0;
  const uint32_t e0 = sampo_f2bits(0x1p-40f), e1 = sampo_f2bits(2.2f), p0 = sampo_f2bits(0.15f), p1 = sampo_f2bits(1.0f);
#pragma omp parallel for schedule(static) reduction(max : ee) reduction(+ : ef, em, en)
  for (long long j = e0; j < (long long)e1; j += stride) {
    const float x = sampo_bits2f((uint32_t)j);
    float H, L, f;
    en++;
    if (sampo_exp_pair(x, 0.0f, &H, &L)) {
      const double ref = exp((double)x), rel = fabs(((double)H + (double)L) - ref) / ref;
      if (rel > ee) ee = rel;
      if (!sampo_round_test(H, L, SAMPO_FAST_EXP_EPS, &f)) ef++;
    } else {
      ef++;
    }
    if (sampo_f2bits(sampo_expf_hourly(x)) != sampo_f2bits(sampo_expf(x))) em++;
  }
#pragma omp parallel for schedule(static) reduction(max : pe) reduction(+ : pf, pm, pn)
  for (long long j = p0; j < (long long)p1; j += stride) {
    const float x = sampo_bits2f((uint32_t)j), y = 1.0f / 24.0f;
    float h, l, H, L, f;
    pn++;
    if (sampo_log_pair(x, &h, &l)) {
      const float zh = y * h, zl = sampo_fmaf(y, h, -zh) + y * l;
      if (sampo_exp_pair(zh, zl, &H, &L)) {
        const double ref = exp((double)y * log((double)x)), rel = fabs(((double)H + (double)L) - ref) / ref;
        if (rel > pe) pe = rel;
        if (!sampo_round_test(H, L, SAMPO_FAST_POW_EPS, &f)) pf++;
      } else {
        pf++;
      }
    }
    if (sampo_f2bits(sampo_powf_hourly(x)) != sampo_f2bits(sampo_powf(x, y))) pm++;
  }
  const float special[] = {0.0f, -0.0f, 0x1p-149f, 0x1p-126f, 2.2f, 2.0794415f, 2.0794416f, 2.0794418f, 3.0f, 88.7f, 89.0f, 1e30f, INFINITY, NAN};
  for (size_t k = 0; k < sizeof(special) / sizeof(special[0]); k++)
    if (sampo_f2bits(sampo_larva_hmr(special[k])) != sampo_f2bits(hmr_definition(special[k]))) hm++;
  const uint32_t h1 = sampo_f2bits(4.0f);
#pragma omp parallel for schedule(static) reduction(+ : hm)
  for (long long j = e0; j < (long long)h1; j += 4 * (long long)stride + 1) {
    const float x = sampo_bits2f((uint32_t)j);
    if (sampo_f2bits(sampo_larva_hmr(x)) != sampo_f2bits(hmr_definition(x))) hm++;
  }
  printf("exp n=%lld maxrel=2^%.2f fallbacks=%lld mismatches=%lld\n", en, log2(ee), ef, em);
  printf("pow n=%lld maxrel=2^%.2f fallbacks=%lld mismatches=%lld\n", pn, log2(pe), pf, pm);
  printf("hmr mismatches=%lld\n", hm);
  return em || pm || hm ? 1 : 0;
}
