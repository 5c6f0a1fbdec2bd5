// Host run of the streamwise lines (csrc/xpass.cuh) and of the two-butterfly
// lines (csrc/zpass.cuh plans, as csrc/xline.cuh takes them): every pass
// butterfly by butterfly with the device's index arithmetic and tables, compared
// with a long-double DFT, and every twiddle with its exact value.  Built and run
// by tests/test_xpass_host.py.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "../../gpu-spectral-channel-dns_b200/csrc/xpass.cuh"
#include "../../gpu-spectral-channel-dns_b200/csrc/zpass.cuh"

static const long double PI = 3.141592653589793238462643383279502884L;

template <typename C> double distance(C a, int j, int L) {
  const long double x = -2 * PI * (j % L) / L;
  return (double)hypotl(a.x - cosl(x), a.y - sinl(x));
}

// the passes of a radix list on one padded line; tw_err: worst twiddle
template <typename C, int L, bool INV, int Ns, int TWO, int R, int... Rest>
void passes(std::vector<C>& line, const C* tw, double& tw_err) {
  typedef XPass<C, L, R, Ns, TWO, INV> P;
  std::vector<C> v((size_t)P::NB * R);
  for (int j = 0; j < P::NB; ++j) {
    C w[R];
    if (Ns > 1) {
      P::weights(tw, j, w);
      for (int r = 1; r < R; ++r) tw_err = fmax(tw_err, distance(w[r], r * (j % Ns) * (L / (Ns * R)), L));
    }
    P::load(line.data(), j, &v[(size_t)j * R]);
    P::run(&v[(size_t)j * R], w);
  }
  for (int j = 0; j < P::NB; ++j) P::store(line.data(), j, &v[(size_t)j * R]);
  if constexpr (sizeof...(Rest) > 0)
    passes<C, L, INV, Ns * R, TWO + (Ns > 1 ? (R - 1) * Ns : 0), Rest...>(line, tw, tw_err);
}
template <typename C, int L, bool INV, int... Rs> void all(Radices<Rs...>, std::vector<C>& line, const C* tw, double& e) {
  passes<C, L, INV, 1, 0, Rs...>(line, tw, e);
}

template <typename C, int L> std::vector<C> input() {
  std::mt19937 rng(L * 11 + 3);
  std::normal_distribution<double> nd;
  std::vector<C> x(L);
  for (C& v : x) v = cmk<C>(nd(rng), nd(rng));
  return x;
}
template <typename C, int L> double error(const std::vector<C>& in, const std::vector<C>& line, bool inv) {
  double err = 0, nrm = 0;
  std::vector<long double> ct(L), st(L);
  for (int n = 0; n < L; ++n) {
    ct[n] = cosl(2 * PI * n / L);
    st[n] = (inv ? 1 : -1) * sinl(2 * PI * n / L);
  }
  for (int k = 0; k < L; ++k) {
    long double sr = 0, si = 0;
    for (int n = 0; n < L; ++n) {
      const long double c = ct[(long long)n * k % L], s = st[(long long)n * k % L];
      sr += in[n].x * c - in[n].y * s;
      si += in[n].x * s + in[n].y * c;
    }
    const C got = line[wsw<C>(k)];
    err = fmax(err, (double)hypotl(got.x - sr, got.y - si));
    nrm = fmax(nrm, (double)hypotl(sr, si));
  }
  return err / nrm;
}
template <typename C, int L> std::vector<C> padded(const std::vector<C>& in) {
  std::vector<C> line(wlen<C>(L) + 1, cmk<C>(1e30, 1e30));
  for (int n = 0; n < L; ++n) line[wsw<C>(n)] = in[n];
  return line;
}
template <int L> std::vector<double2> base_table() {
  std::vector<double2> W(L);
  for (int j = 0; j < L; ++j) W[j] = make_double2((double)cosl(-2 * PI * j / L), (double)sinl(-2 * PI * j / L));
  return W;
}

template <typename C, int L> void stream(const char* name) {
  typedef XPlan<L, FftMaxRadix<C>::v> P;
  std::vector<C> tw;
  xtw_table<C>(L, base_table<L>().data(), tw);
  const std::vector<C> in = input<C, L>();
  double te = 0;
  std::vector<C> a = padded<C, L>(in), b = a;
  all<C, L, true>(typename P::INV(), a, tw.data(), te);
  all<C, L, false>(typename P::FWD(), b, tw.data() + wtw_size(typename P::INV()), te);
  printf("stream %s %d %.3e %.3e %.3e\n", name, L, te, error<C, L>(in, a, true), error<C, L>(in, b, false));
}

template <typename C, int L, bool INV> double two(double& te) {
  constexpr int A = ZPlan<L>::A, B = ZPlan<L>::B;
  typedef XPass<C, L, A, 1, 0, INV> PA;
  typedef XPass<C, L, B, A, 0, INV> PB;
  std::vector<C> tw;
  ztw_table<C>(L, base_table<L>().data(), tw);
  const std::vector<C> in = input<C, L>();
  std::vector<C> line = padded<C, L>(in), v((size_t)L);
  for (int j = 0; j < B; ++j) {
    PA::load(line.data(), j, &v[(size_t)j * A]);
    PA::run(&v[(size_t)j * A], nullptr);
  }
  for (int j = 0; j < B; ++j) PA::store(line.data(), j, &v[(size_t)j * A]);
  for (int k = 0; k < A; ++k) {
    C w[B];
    for (int r = 1; r < B; ++r) {
      w[r] = tw[(r - 1) * A + k];
      te = fmax(te, distance(w[r], r * k, L));
    }
    PB::load(line.data(), k, &v[(size_t)k * B]);
    PB::run(&v[(size_t)k * B], w);
  }
  for (int k = 0; k < A; ++k) PB::store(line.data(), k, &v[(size_t)k * B]);
  return error<C, L>(in, line, INV);
}
template <typename C, int L> void span(const char* name) {
  double te = 0;
  const double ei = two<C, L, true>(te), ef = two<C, L, false>(te);
  printf("span %s %d %.3e %.3e %.3e\n", name, L, te, ei, ef);
}

int main() {
#define XC(n) stream<float2, n>("float2"); stream<double2, n>("double2");
#define ZC(n) span<float2, n>("float2"); span<double2, n>("double2");
  XPLAN_LENGTHS(XC)
  ZPLAN_LENGTHS(ZC)
  return 0;
}
