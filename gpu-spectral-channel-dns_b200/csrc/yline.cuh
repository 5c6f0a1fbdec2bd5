// Device helpers of the wall-normal kernels (ypass.cu, ystep.cuh).
#pragma once
#include "kernels.cuh"

namespace {

struct Carve {
  char* p;
  __device__ explicit Carve(void* b) : p((char*)b) {}
  template <class T> __device__ T* take(size_t n) {
    T* r = (T*)p;
    p += (n * sizeof(T) + 15) & ~(size_t)15;
    return r;
  }
};

// Chebyshev coefficient derivative executed by one full warp:
// b_i = sum_{j>i, j-i odd} 2 j a_j, b_0 halved (source/RPCFKernels.cu:476-520),
// evaluated as parity-split suffix sums.  a, b in shared memory, no alias.
__device__ __noinline__ void ddz_warp(const double2* a, double2* b, int N) {
  const int lane = threadIdx.x & 31;
  const int c = (N + 31) / 32;
  const int j0 = lane * c;
  const int j1 = min(j0 + c, N);
  double er = 0, ei = 0, orr = 0, oi = 0;
  for (int j = j0; j < j1; ++j) {
    double2 v = a[j];
    double f = 2.0 * j;
    if (j & 1) { orr += f * v.x; oi += f * v.y; }
    else { er += f * v.x; ei += f * v.y; }
  }
  double s0 = er, s1 = ei, s2 = orr, s3 = oi;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    double t0 = __shfl_down_sync(0xffffffffu, s0, d);
    double t1 = __shfl_down_sync(0xffffffffu, s1, d);
    double t2 = __shfl_down_sync(0xffffffffu, s2, d);
    double t3 = __shfl_down_sync(0xffffffffu, s3, d);
    if (lane + d < 32) { s0 += t0; s1 += t1; s2 += t2; s3 += t3; }
  }
  double re_e = s0 - er, im_e = s1 - ei, re_o = s2 - orr, im_o = s3 - oi;
  for (int j = j1 - 1; j >= j0; --j) {
    double2 v = a[j];
    double f = 2.0 * j;
    double2 out = (j & 1) ? make_double2(re_e, im_e) : make_double2(re_o, im_o);
    if (j == 0) out = out * 0.5;
    b[j] = out;
    if (j & 1) { re_o += f * v.x; im_o += f * v.y; }
    else { re_e += f * v.x; im_e += f * v.y; }
  }
}

// The same derivative with CH (even) coefficients per lane: every lane's
// run starts at an even index, so the parity of each of its elements is
// known at compile time (the sums split by parity without divergent
// branches), and the run stays in registers between the two sweeps.  E is
// the element type: double2, or float2 where the result feeds FP32
// transforms only.
template <int CH, typename E = double2>
__device__ __noinline__ void ddz_fast(const E* __restrict__ a, E* __restrict__ b, int N) {
  static_assert(CH % 2 == 0, "runs of even length");
  typedef T_of<E> S;
  const int lane = threadIdx.x & 31;
  const int j0 = lane * CH;
  E v[CH];
#pragma unroll
  for (int i = 0; i < CH; ++i) v[i] = (j0 + i < N) ? a[j0 + i] : cmk<E>(0.0, 0.0);
  E te = cmk<E>(0.0, 0.0), to = te;  // this run's sums of 2 j a_j, even / odd j
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const S f = (S)(2 * (j0 + i));
    if (i & 1) to = to + v[i] * f;
    else te = te + v[i] * f;
  }
  S s0 = te.x, s1 = te.y, s2 = to.x, s3 = to.y;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const S t0 = __shfl_down_sync(0xffffffffu, s0, d);
    const S t1 = __shfl_down_sync(0xffffffffu, s1, d);
    const S t2 = __shfl_down_sync(0xffffffffu, s2, d);
    const S t3 = __shfl_down_sync(0xffffffffu, s3, d);
    if (lane + d < 32) { s0 += t0; s1 += t1; s2 += t2; s3 += t3; }
  }
  // sums over the runs of the lanes above, then down this run
  E re = cmk<E>(s0 - te.x, s1 - te.y), ro = cmk<E>(s2 - to.x, s3 - to.y);
#pragma unroll
  for (int i = CH - 1; i >= 0; --i) {
    const int j = j0 + i;
    E out = (i & 1) ? re : ro;  // j' > j of the other parity
    if (j == 0) out = out * (S)0.5;
    if (j < N) b[j] = out;
    const S f = (S)(2 * j);
    if (i & 1) ro = ro + v[i] * f;
    else re = re + v[i] * f;
  }
}

// even extension for the padded s2p (cheby_pre_s2p_pad): e[0] = c0,
// e[k] = e[M-k] = c_k/2 for 1 <= k <= Ny-1, zero otherwise; M = 4(Ny-1).
template <typename C>
__device__ __forceinline__ double2 ext_s2p_pad(const double2* c, int n, int M, int Ny) {
  if (n == 0) return c[0];
  if (n <= Ny - 1) return c[n] * 0.5;
  if (n >= M - (Ny - 1)) return c[M - n] * 0.5;
  return make_double2(0.0, 0.0);
}

template <typename C>
__device__ __forceinline__ C* pencil_ptr(const PencilArr& a, int f, long long p) {
  return (C*)a.base + (long long)f * a.fs + p * a.ps;
}

}  // namespace
