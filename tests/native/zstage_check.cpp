// Host check of the tensor-staged spanwise tiles (csrc/zpass.cuh): where every
// tensor copy of a length lands in shared memory, against the rules of tiled
// copies.  Built and run by tests/test_span_stage_host.py.
#include <cstdio>

#include "../../gpu-spectral-channel-dns_b200/csrc/zpass.cuh"

template <int L> void forward() {
  typedef ZStage<float2, L> Z;
  const bool taken = Z::ok && Z::fits(L) && Z::copies_ok;
  // length, taken, bytes of the pair, then per copy: first row, rows, byte
  // offset of its destination from the tile (elements as in k_zft)
  printf("%d %d %d", L, (int)taken, Z::WS * (int)sizeof(float2));
  if (taken)
    for (int z = 0; z < L; z += Z::ROWS) printf(" %d %d %d", z, Z::ROWS, 2 * z * (int)sizeof(float2));
  printf("\n");
}

int main() {
#define CASE(n) forward<n>();
  ZPLAN_LENGTHS(CASE)
  return 0;
}
