/* Exhaustive check of the two-operation x / 3 that the GPU's Jarosz kernel uses for the sums
 * of byte images (div3 in yume-pdq_gb300/csrc/jarosz.cu): RN(x c + RN(x c')) with c = RN(1/3)
 * and c' = RN(1/3 - c), against IEEE x / 3 for zero and every finite positive float from
 * 2^-120 on (each step is odd in x). Built with -ffp-contract=off. */
#include <math.h>
#include <pthread.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

enum { kThreads = 8 };

typedef struct {
  uint64_t lo, hi, bad;
} job;

static float as_float(uint32_t b) {
  float x;
  memcpy(&x, &b, 4);
  return x;
}

static void* run(void* p) {
  job* j = (job*)p;
  for (uint64_t b = j->lo; b < j->hi; b++) {
    const float x = as_float((uint32_t)b);
    const float q = fmaf(x, 0x1.555556p-2f, x * -0x1.555556p-27f), want = x / 3.0f;
    j->bad += memcmp(&q, &want, 4) != 0;
  }
  return NULL;
}

int main(void) {
  const uint64_t lo = (uint64_t)(127 - 120) << 23, hi = (uint64_t)255 << 23;
  pthread_t th[kThreads];
  job jobs[kThreads];
  uint64_t bad = 0;
  const float zero = fmaf(0.0f, 0x1.555556p-2f, 0.0f * -0x1.555556p-27f);
  if ((float)(1.0L / 3 - (long double)0x1.555556p-2f) != -0x1.555556p-27f) {
    printf("RN(1/3 - RN(1/3)) constant wrong\n");
    return 2;
  }
  for (int i = 0; i < kThreads; i++) {
    jobs[i] = (job){lo + (hi - lo) * i / kThreads, lo + (hi - lo) * (i + 1) / kThreads, 0};
    pthread_create(&th[i], NULL, run, &jobs[i]);
  }
  for (int i = 0; i < kThreads; i++) {
    pthread_join(th[i], NULL);
    bad += jobs[i].bad;
  }
  printf("mismatches %llu\n", (unsigned long long)bad);
  return bad != 0 || zero != 0.0f;
}
