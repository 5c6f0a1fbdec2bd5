// Chebyshev-coefficient helpers of the wall-normal kernels.
#pragma once
#include "kernels.cuh"

// Sums over the 16 lanes of a parity of NV values a lane, the values halved
// between a lane and its partner at every step (masks 16, 8, 4, 2; 11 exchanges
// for ten values instead of 40).  Where an odd count is halved the upper lane
// gets one fewer, so that some lanes end with none.
template <int NV> struct ParitySums {
  enum { HALF = (NV + 1) / 2 };
  // a step on n values, the first (n + 1) / 2 to the lower lane: v keeps the
  // lane's own, send goes to the partner
  DNS_HD static void split(double (&v)[NV], double (&send)[HALF], int n, bool up) {
    const int half = (n + 1) / 2;
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      if (i >= half) continue;
      const double hi = i + half < n ? v[i + half] : 0.0;
      send[i] = up ? v[i] : hi;
      v[i] = up ? hi : v[i];
    }
  }
  // the value whose sum the lane ends with, NV: none
  DNS_HD static int slot(int lane) {
    int idx = 0, cnt = NV;  // this lane's values idx .. idx + cnt - 1
#pragma unroll
    for (int m = 16, n = NV; m > 1; m >>= 1) {
      const int half = (n + 1) / 2;
      if (lane & m) {
        idx += half;
        cnt -= half;
      } else if (cnt > half) {
        cnt = half;
      }
      n = half;
    }
    return cnt > 0 ? idx : (int)NV;
  }
#ifdef __CUDACC__
  __device__ __forceinline__ static double run(double (&v)[NV], int lane) {
    int n = NV;
#pragma unroll
    for (int m = 16; m > 1; m >>= 1) {
      double send[HALF];
      split(v, send, n, lane & m);
      n = (n + 1) / 2;
#pragma unroll
      for (int i = 0; i < HALF; ++i)
        if (i < n) v[i] += __shfl_xor_sync(0xffffffffu, send[i], m);
    }
    return v[0];
  }
#endif
};

#ifdef __CUDACC__

// run length of a lane for Ny coefficients (even: the parity of each of its
// elements is known at compile time)
__host__ __device__ constexpr int ddz_run(int Ny) { return 2 * ((Ny + 63) / 64); }

// coefficient k of U X and, for k <= N, of its Gauss-Lobatto interpolant
// (degrees N + 1, N + 2 fold to N - 1, N - 2); X has two zeros below 0 and two
// above N
__device__ __forceinline__ void u_times(const double2* X, int k, int N, const PhysParams& ph, double2& P, double2& Pf) {
  P = X[k] * ph.U0 + (X[k - 1] * (k == 1 ? 1.0 : 0.5) + X[k + 1] * 0.5) * ph.U1;
  if (ph.U2 != 0.0)
    P = P + (X[k - 2] * (k == 2 ? 0.5 : 0.25) + X[k] * (k == 1 ? 0.75 : 0.5) + X[k + 2] * 0.25) * ph.U2;
  Pf = P;
  if (k == N - 1) Pf = Pf + X[N] * (0.5 * ph.U1) + X[N - 1] * (0.25 * ph.U2);
  if (k == N - 2) Pf = Pf + X[N] * (0.25 * ph.U2);
}
// coefficient k <= N of the interpolant of U' X
__device__ __forceinline__ double2 up_times(const double2* X, int k, int N, const PhysParams& ph) {
  double2 r = X[k] * ph.U1;
  if (ph.U2 != 0.0) {
    r = r + (X[k - 1] * (k == 1 ? 2.0 : 1.0) + X[k + 1]) * ph.U2;
    if (k == N - 1) r = r + X[N] * ph.U2;
  }
  return r;
}

// Second derivative of a Chebyshev series by one warp in one sweep, CH
// (even) coefficients per lane: b_i = (1 / c_i) sum_{j >= i+2, j - i even}
// j (j^2 - i^2) a_j (c_0 = 2, else 1), as parity-split suffix sums of j a_j
// and j^3 a_j.
template <int CH>
__device__ __noinline__ void d2z_fast(const double2* __restrict__ a, double2* __restrict__ b, int N) {
  static_assert(CH % 2 == 0, "runs of even length");
  const int lane = threadIdx.x & 31;
  const int j0 = lane * CH;
  double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // (j a_j, j^3 a_j) x (even, odd j), re / im
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    if (j0 + i < N) {
      const double2 v = a[j0 + i];
      const double j = (double)(j0 + i), j3 = j * j * j;
      const int o = (i & 1) * 4;
      t[o + 0] += j * v.x;
      t[o + 1] += j * v.y;
      t[o + 2] += j3 * v.x;
      t[o + 3] += j3 * v.y;
    }
  }
  // inclusive suffix sums over the lanes, then those of the lanes above
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double x = __shfl_down_sync(0xffffffffu, t[k], d);
      if (lane + d < 32) t[k] += x;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double x = __shfl_down_sync(0xffffffffu, t[k], 1);
    t[k] = lane < 31 ? x : 0.0;
  }
#pragma unroll
  for (int i = CH - 1; i >= 0; --i) {
    const int jj = j0 + i;
    if (jj < N) {
      const double j = (double)jj, j2 = j * j;
      const int o = (i & 1) * 4;  // j' >= j + 2 of the same parity
      double2 out = make_double2(t[o + 2] - j2 * t[o + 0], t[o + 3] - j2 * t[o + 1]);
      if (jj == 0) out = out * 0.5;
      const double2 v = a[jj];
      b[jj] = out;
      t[o + 0] += j * v.x;
      t[o + 1] += j * v.y;
      t[o + 2] += j * j2 * v.x;
      t[o + 3] += j * j2 * v.y;
    }
  }
}
#endif
