// crand_unit against the division it stands for: the first and last million
// numerators, every power of two with its neighbours, and a stride through
// the rest.  Prints the number of differences.
#include <cstdio>

#include "../mcgpu_gb300/csrc/crand.h"

int main() {
  const long long top = 2147483647LL;
  long long bad = 0;
  auto check = [&](long long v) {
    if (v < 0 || v > top) return;
    if (mcgpu::crand_unit((int32_t)v) != (double)v / 2147483647.0) bad++;
  };
  for (long long v = 0; v < 1000000; v++) {
    check(v);
    check(top - v);
  }
  for (int k = 0; k < 31; k++)
    for (int d = -2; d <= 2; d++) check((1LL << k) + d);
  for (long long v = 17; v <= top; v += 1009) check(v);
  printf("%lld\n", bad);
  return 0;
}
