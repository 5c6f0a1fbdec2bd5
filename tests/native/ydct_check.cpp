// Host run of the pruned DCT (csrc/ydct.cuh): both passes butterfly by
// butterfly with the device's index arithmetic, compared with a long-double
// DFT of the even extension.  Built and run by tests/test_dct_host.py.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "../../gpu-spectral-channel-dns_b200/csrc/ydct.cuh"

template <typename C, int M, int NL, int N0> double check() {
  const long double PI = 3.141592653589793238462643383279502884L;
  typedef Dct<C, M, NL> D;
  constexpr int H = M / 2;
  std::mt19937 rng(M * 5 + NL + N0);
  std::normal_distribution<double> nd;
  std::vector<C> e(NL * (H + 1)), X(D::XN, cmk<C>(1e30, 1e30)), out(NL * (H + 1), cmk<C>(1e30, 1e30)), tw;
  for (int l = 0; l < NL; ++l)
    for (int n = 0; n <= H; ++n) e[l * (H + 1) + n] = (N0 && n >= N0) ? cmk<C>(0.0, 0.0) : cmk<C>(nd(rng), nd(rng));
  std::vector<double2> W(M);
  for (int j = 0; j < M; ++j) W[j] = make_double2((double)cosl(-2 * PI * j / M), (double)sinl(-2 * PI * j / M));
  dtw_table<C>(M, W.data(), tw);
  for (int i = 0; i < D::IA; ++i)
    D::template pass_a<N0>(X.data(), i, [&](int l, int n) { return e[l * (H + 1) + n]; });
  for (int i = 0; i < D::IB; ++i)
    D::pass_b(X.data(), tw.data(), i, [&](int l, int k, C v) { out[l * (H + 1) + k] = v; });
  double err = 0, nrm = 0;
  for (int l = 0; l < NL; ++l)
    for (int k = 0; k <= H; ++k) {
      long double sr = 0, si = 0;
      for (int n = 0; n < M; ++n) {
        const C v = e[l * (H + 1) + (n <= H ? n : M - n)];
        const long double c = cosl(2 * PI * (long double)((long long)n * k % M) / M);
        sr += v.x * c;
        si += v.y * c;
      }
      const C got = out[l * (H + 1) + k];
      err = fmax(err, (double)hypotl(got.x - sr, got.y - si));
      nrm = fmax(nrm, (double)hypotl(sr, si));
    }
  return err / nrm;
}

#define CASE(M)                                                                                                   \
  printf("float2 %d %.3e %.3e %.3e\n", M, check<float2, M, 6, M / 4 + 1>(), check<float2, M, 3, 0>(),             \
         check<float2, M, 1, 0>());                                                                               \
  printf("double2 %d %.3e %.3e %.3e\n", M, check<double2, M, 6, M / 4 + 1>(), check<double2, M, 3, 0>(),          \
         check<double2, M, 1, 0>());

int main() {
  DPLAN_SHORT(CASE)
  DPLAN_LENGTHS(CASE)
  return 0;
}
