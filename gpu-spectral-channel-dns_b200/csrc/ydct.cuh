// Chebyshev (DCT-I) transforms as pruned FFTs of the even extension.
//
// The line e[n], n < M, is even (e[M - n] = e[n]), and so is its transform E.
// M = RA RB, two passes: pass A takes X_j[s] = sum_r e[j + r RB] W_RA^{r s}
// for j = 0 .. RB/2 only, since X_{RB-j}[s] = W_RA^{-s} X_j[-s]; pass B takes
// E[s + t RA] = sum_j (W_M^{j s} X_j[s]) W_RB^{j t} for s = 0 .. RA/2 only,
// since E[M - k] = E[k], with W_M^{(RB-j) s} X_{RB-j}[s] = conj(W_M^{j s})
// X_j[RA - s].  So both passes do little more than half the butterflies of
// the whole FFT (9 of 16 and 17 of 32 at M = 512), at the FFT's accuracy: no
// prefix sums, no division by sines.
#pragma once
#include <type_traits>
#include <vector>

#include "fft2.cuh"
#include "kernels.cuh"

// index range hints (resolve, per compile-time r, which branch of a load or
// store applies)
#ifdef __CUDA_ARCH__
#define YDCT_ASSUME(c) __builtin_assume(c)
#else
#define YDCT_ASSUME(c) ((void)0)
#endif

template <int M> struct DPlan { enum { ok = 0, A = 2, B = 2 }; };
#define DPLAN(M, RA, RB)                                                                      \
  template <> struct DPlan<M> {                                                               \
    enum { ok = 1, A = RA, B = RB };                                                          \
    static_assert(RA * RB == M && RA % 2 == 0 && RB % 2 == 0 && M % 4 == 0, "plan");          \
  };
DPLAN(16, 4, 4)
DPLAN(24, 6, 4)
DPLAN(32, 8, 4)
DPLAN(36, 6, 6)
DPLAN(48, 8, 6)
DPLAN(64, 8, 8)
DPLAN(72, 12, 6)
DPLAN(96, 12, 8)
DPLAN(108, 18, 6)
DPLAN(128, 16, 8)
DPLAN(144, 12, 12)
DPLAN(192, 16, 12)
DPLAN(216, 18, 12)
DPLAN(256, 16, 16)
DPLAN(288, 18, 16)
DPLAN(324, 18, 18)
DPLAN(384, 24, 16)
DPLAN(432, 24, 18)
DPLAN(512, 32, 16)
DPLAN(576, 32, 18)
DPLAN(768, 32, 24)
#undef DPLAN
#define DPLAN_LENGTHS(X) \
  X(32) X(36) X(48) X(64) X(72) X(96) X(108) X(128) X(144) X(192) X(216) X(256) X(288) X(324) X(384) X(432) \
  X(512) X(576) X(768)

// lengths of the no-padding transforms only
#define DPLAN_SHORT(X) X(16) X(24)

// Elements of the derivatives in getUVW.  The mixed form rounds the state to
// FP32 first at the lengths below, where it always did; at the others the sweeps
// are FP64, as in the block form, and only the six fields are rounded.
template <typename C, int M> struct Y3Form {
  static constexpr bool fp32 = sizeof(C) == 8 && (M == 128 || M == 192 || M == 256 || M == 384 || M == 512 || M == 768);
  typedef typename std::conditional<fp32, float2, double2>::type E;
};

// pass-B twiddles W_M^{j s}, j = 1..RB/2, s = 0..RA/2, stored [j - 1][s]; W:
// the table W_M^j, j < M
template <typename C> int dtw_table(int M, const double2* W, std::vector<C>& out) {
  int ra = 0, rb = 0;
#define DCASE(n) \
  case n: ra = DPlan<n>::A; rb = DPlan<n>::B; break;
  switch (M) { DPLAN_SHORT(DCASE) DPLAN_LENGTHS(DCASE) default: return -1; }
#undef DCASE
  const int sh = ra / 2 + 1;
  out.resize((size_t)(rb / 2) * sh);
  for (int j = 1; j <= rb / 2; ++j)
    for (int s = 0; s < sh; ++s) out[(size_t)(j - 1) * sh + s] = from_d2<C>(W[j * s]);
  return (int)out.size();
}

// NL lines; X: RA rows [s] of XP columns (line JH + j), XP odd: the lanes of
// pass B, consecutive s, fall in distinct banks
template <typename C, int M, int NL> struct Dct {
  static constexpr int RA = DPlan<M>::A, RB = DPlan<M>::B;
  static constexpr int JH = RB / 2 + 1, SH = RA / 2 + 1;
  static constexpr int XP = (NL * JH) | 1;
  static constexpr int XN = RA * XP;            // complex values of X
  static constexpr int IA = NL * JH, IB = NL * SH;  // butterflies of pass A, B
  // butterfly i of pass A; ld(line, n) gives e[n], 0 <= n <= M/2.  n0 > 0:
  // e[n] = 0 for n0 <= n <= M/2
  template <int N0, class LD> DNS_HD static void pass_a(C* X, int i, LD ld) {
    const int l = i / JH, j = i - l * JH;
    YDCT_ASSUME(j >= 0 && j < JH);
    C v[RA];
#pragma unroll
    for (int r = 0; r < RA; ++r) {
      // n = j + r RB, j <= RB/2: folded beyond M/2
      const int n = j + r * RB;
      v[r] = cmk<C>(0.0, 0.0);
      if (2 * r < RA) {  // n <= M/2
        if (N0 == 0 || r * RB < N0) {
          if (N0 == 0 || n < N0) v[r] = ld(l, n);
        }
      } else {           // M - n <= M/2
        if (N0 == 0 || M - (r * RB + RB / 2) < N0) {
          if (N0 == 0 || M - n < N0) v[r] = ld(l, M - n);
        }
      }
    }
    Codelet<RA, false, C>::run(v);
    C* x = X + i;
#pragma unroll
    for (int s = 0; s < RA; ++s) x[s * XP] = v[s];
  }
  // butterfly i of pass B; st(line, k, E[k]) for its outputs, 0 <= k <= M/2
  // (some twice, with equal values)
  template <class ST> DNS_HD static void pass_b(const C* X, const C* tw, int i, ST st) {
    const int l = i / SH, s = i - l * SH;
    YDCT_ASSUME(s >= 0 && s < SH);
    const C* xs = X + s * XP + l * JH;
    const C* xm = X + (s ? RA - s : 0) * XP + l * JH;
    C v[RB];
    v[0] = xs[0];
#pragma unroll
    for (int j = 1; j <= RB / 2; ++j) {
      const C w = tw[(j - 1) * SH + s];
      v[j] = cmul(xs[j], w);
      if (j < RB / 2) v[RB - j] = cmulc(xm[j], w);
    }
    Codelet<RB, false, C>::run(v);
#pragma unroll
    for (int t = 0; t < RB; ++t) {
      const int k = s + t * RA;
      if (2 * t < RB) st(l, k, v[t]);  // k < M/2, or = M/2 by the mirror of t >= RB/2
      else st(l, M - k, v[t]);
    }
  }
};

#define YDCT_CASE(n) case n: return f(std::integral_constant<int, n>());
// the lengths of the time step, and with the short ones of small no-padding
// transforms; cudaErrorNotSupported for others
template <typename F> cudaError_t with_len_d(int M, F&& f) {
  switch (M) { DPLAN_LENGTHS(YDCT_CASE) }
  return cudaErrorNotSupported;
}
template <typename F> cudaError_t with_len_cheby(int M, F&& f) {
  switch (M) { DPLAN_SHORT(YDCT_CASE) DPLAN_LENGTHS(YDCT_CASE) }
  return cudaErrorNotSupported;
}
