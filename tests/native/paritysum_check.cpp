// Host run of the parity sums (csrc/ycoef.cuh): a warp's lanes in step, and
// which of them hold which sum.  Built and run by tests/test_parity_sums_host.py.
#include <cstdio>
#include <vector>

#include "../../gpu-spectral-channel-dns_b200/csrc/ycoef.cuh"

template <int NV> void check() {
  typedef ParitySums<NV> P;
  static double v[32][NV], send[32][P::HALF];
  double want[2][NV] = {};
  for (int l = 0; l < 32; ++l)
    for (int i = 0; i < NV; ++i) {
      v[l][i] = (double)((l * 37 + i * 101 + 13) % 211 + 1);  // whole numbers: the sums are exact
      want[l & 1][i] += v[l][i];
    }
  int n = NV;
  for (int m = 16; m > 1; m >>= 1) {
    for (int l = 0; l < 32; ++l) P::split(v[l], send[l], n, l & m);
    n = (n + 1) / 2;
    for (int l = 0; l < 32; ++l)
      for (int i = 0; i < n; ++i) v[l][i] += send[l ^ m][i];
  }
  int writers[2][NV] = {}, wrong = 0;
  for (int l = 0; l < 32; ++l) {
    const int s = P::slot(l);
    if (s < 0 || s > NV) ++wrong;
    if (s < 0 || s >= NV) continue;
    ++writers[l & 1][s];
    if (v[l][0] != want[l & 1][s]) ++wrong;
  }
  int bad = 0;
  for (int p = 0; p < 2; ++p)
    for (int i = 0; i < NV; ++i) bad += writers[p][i] != 1;
  printf("%d %d %d\n", NV, bad, wrong);
}

int main() {
  check<1>(); check<2>(); check<3>(); check<5>(); check<6>(); check<7>(); check<8>(); check<10>(); check<12>();
  check<13>(); check<16>();
  return 0;
}
