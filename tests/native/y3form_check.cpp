// Element sizes of the getUVW derivatives per length and precision
// (csrc/ydct.cuh).  Built and run by tests/test_y3_form_host.py.
#include <cstdio>

#include "../../gpu-spectral-channel-dns_b200/csrc/ydct.cuh"

int main() {
#define CASE(M) printf("%d %d %d\n", M, (int)sizeof(Y3Form<float2, M>::E), (int)sizeof(Y3Form<double2, M>::E));
  DPLAN_LENGTHS(CASE)
  return 0;
}
