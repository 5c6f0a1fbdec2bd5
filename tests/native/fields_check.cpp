// Host check of which fields of one transform call share launches
// (csrc/kernels.cuh), against a byte-by-byte map.  Built and run by
// tests/test_fields_host.py.
#include <cstdio>
#include <random>
#include <set>

#include "../../gpu-spectral-channel-dns_b200/csrc/kernels.cuh"

static std::set<long long> bytes(const PitchedBytes& a) {
  std::set<long long> s;
  for (long long i = 0; i < a.n; ++i)
    for (long long k = 0; k < a.w; ++k) s.insert((long long)(size_t)a.p + i * a.pitch + k);
  return s;
}
static bool meet(const PitchedBytes& a, const PitchedBytes& b) {
  const std::set<long long> x = bytes(a);
  for (long long v : bytes(b))
    if (x.count(v)) return true;
  return false;
}

int main() {
  // rows of one pitch and of two, at every distance: never "apart" where a byte is shared
  std::mt19937 rng(3);
  int missed = 0, cases = 0;
  for (int t = 0; t < 20000; ++t) {
    auto in = [&](int lo, int hi) { return (long long)(lo + (int)(rng() % (unsigned)(hi - lo + 1))); };
    const long long pa = in(4, 12), pb = t & 1 ? pa : in(4, 12);
    const PitchedBytes a{(void*)(size_t)in(100, 160), in(1, 5), in(1, (int)pa), pa};
    const PitchedBytes b{(void*)(size_t)in(100, 160), in(1, 5), in(1, (int)pb), pb};
    const bool want = meet(a, b), got = rows_overlap(a, b);
    if (want && !got) ++missed;
    if (want != rows_overlap(b, a) && want) ++missed;
    ++cases;
  }
  printf("random %d %d\n", cases, missed);
  // fields as a caller lays them out: 4 rows of 16 bytes of points, 3 of 32 of pencils
  auto ph = [](size_t p) { return PitchedBytes{(void*)p, 4, 16, 16}; };
  auto sp = [](size_t p) { return PitchedBytes{(void*)p, 3, 32, 32}; };
  const PitchedBytes P[3] = {ph(1000), ph(1064), ph(1128)}, S[3] = {sp(2000), sp(2096), sp(2192)};
  printf("apart %d %d\n", fields_apart(false, 3, P, S), fields_apart(true, 3, P, S));
  const PitchedBytes Pd[3] = {P[0], P[1], P[1]}, Sd[3] = {S[0], S[1], S[0]};
  printf("same_points %d %d\n", fields_apart(false, 3, Pd, S), fields_apart(true, 3, Pd, S));
  printf("same_pencils %d %d\n", fields_apart(false, 3, P, Sd), fields_apart(true, 3, P, Sd));
  const PitchedBytes Pi[3] = {ph(2000), ph(2096), ph(2192)}, Pn[3] = {ph(2096), P[1], P[2]};
  printf("in_place %d %d\n", fields_apart(false, 3, Pi, S), fields_apart(true, 3, Pi, S));
  printf("next_pencils %d %d\n", fields_apart(false, 3, Pn, S), fields_apart(true, 3, Pn, S));
  // rows interleaved in one allocation
  const PitchedBytes Sl[2] = {{(void*)2000, 3, 32, 64}, {(void*)2032, 3, 32, 64}};
  printf("interleaved %d %d\n", fields_apart(false, 2, P, Sl), fields_apart(true, 2, P, Sl));
  return 0;
}
