/* Check of the client quantizer's float form with a truncating fused
 * multiply-add, trunc(|x| * scale + 0.5 rounded toward zero), against the
 * oracle's integer restatement (d_CQ_IABS_4), for lossy words down to zero,
 * where no separate test for small words is made.  The sum is rounded toward
 * zero, so it never passes the integer above the exact value.
 * Test infrastructure only: links the CPU oracle.
 *
 * Build: gcc -O2 -fopenmp -frounding-math -ffp-contract=off cq_trunc_check.c -lm -L<oracle> -lcortado_oracle
 * Usage: cq_trunc_check <eb_e> <stride>
 * Prints checked and mismatching counts; exit status 1 on any mismatch. */
#include <fenv.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

uint32_t ora_cq(uint32_t v, int eb_e);

static float f_of(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  const int eb_e = atoi(argv[1]);
  const long long stride = atoll(argv[2]);
  const uint32_t thr_bits = (uint32_t)(eb_e + 24) << 23;
  const float sc = f_of((uint32_t)(253 - eb_e) << 23); /* 2^(126 - eb_e) */
  long long checked = 0, bad = 0;
#pragma omp parallel reduction(+ : checked, bad)
  {
    fesetround(FE_TOWARDZERO); /* per thread */
#pragma omp for schedule(static)
    for (long long i = 0; i < (1ll << 32); i += stride) {
      const uint32_t v = (uint32_t)i;
      if ((v & 0x7fffffffu) >= thr_bits) continue;
      const float s = fmaf(f_of(v), sc, f_of((v & 0x80000000u) | 0x3f000000u));
      checked++;
      if ((uint32_t)(int32_t)s != ora_cq(v, eb_e)) bad++; /* C's conversion truncates */
    }
  }
  printf("%lld %lld\n", checked, bad);
  return bad ? 1 : 0;
}
