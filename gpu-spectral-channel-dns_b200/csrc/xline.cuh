// Streamwise lines of the reference-layout transforms (FP64): half spectra
// -> rows of points and back, two rows a complex line.
//
// Two register butterflies around one exchange (the radices of the spanwise
// plan): pass A reads its inputs straight from global memory, consecutive
// lanes consecutive bins or points; the inverse stores its points straight
// from pass B.  The forward transform returns the line to shared memory, where
// a butterfly's inputs were, and unpacks the bins that the spanwise pass
// reads.  Both replace a radix-4 transform of runtime length, one barrier and
// one trip through shared memory per radix: see launch_x_c2r.
#pragma once
#include "xpass.cuh"
#include "zpass.cuh"

template <int L> struct XLine {
  enum {
    A = ZPlan<L>::A, B = ZPlan<L>::B,
    NL = B <= 64 ? 64 / B : 1,                // lines per CTA: one round of pass A
    LS = L + (L >> WSwz<double2>::S) + 1,     // padded line
    MB = A > 24 ? 5 : 8                       // CTAs per SM
  };
};

template <int L>
__global__ void __launch_bounds__(64, XLine<L>::MB) k_c2r2(RowArr in, FieldList out, long long rps, long long nrows,
                                                           const double2* __restrict__ tw) {
  typedef XLine<L> P;
  typedef XPass<double2, L, P::A, 1, 0, true> PA;
  typedef XPass<double2, L, P::B, P::A, 0, true> PB;
  constexpr int hx = L / 3;  // Nx / 2 (the launcher checks it): Nyquist and padding are zero
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* z = (double2*)smem_raw;
  const double2* src = (const double2*)in.base + (long long)blockIdx.y * in.fs;
  const long long r0 = (long long)blockIdx.x * (2 * P::NL);
  for (int i = threadIdx.x; i < P::NL * P::B; i += 64) {
    const int q = i / P::B, j = i - q * P::B;
    WFFT_ASSUME(j >= 0 && j < P::B);
    const long long ra = r0 + 2 * q;
    const bool oka = ra < nrows, okb = ra + 1 < nrows;
    const double2 *a = src + ra * in.rs, *b = a + in.rs;
    double2 v[P::A], av[P::A], bv[P::A];
#pragma unroll
    for (int r = 0; r < P::A; ++r) {
      const int n = j + r * P::B;
      av[r] = bv[r] = make_double2(0.0, 0.0);
      const int k = n < hx ? n : (n > L - hx ? L - n : -1);
      if (k >= 0 && oka) av[r] = a[k];
      if (k >= 0 && okb) bv[r] = b[k];
    }
#pragma unroll
    for (int r = 0; r < P::A; ++r) {
      const int n = j + r * P::B;
      // a + i b, conj(a) + i conj(b) above; the DC bins' imaginary parts are dropped
      if (n == 0) v[r] = make_double2(av[r].x, bv[r].x);
      else if (n < hx) v[r] = make_double2(av[r].x - bv[r].y, av[r].y + bv[r].x);
      else v[r] = make_double2(av[r].x + bv[r].y, bv[r].x - av[r].y);
    }
    PA::run(v, nullptr);
    PA::store(z + q * P::LS, j, v);
  }
  __syncthreads();
  double* dst = (double*)out.p[blockIdx.y];
  for (int i = threadIdx.x; i < P::NL * P::A; i += 64) {
    const int q = i / P::A, k = i - q * P::A;
    WFFT_ASSUME(k >= 0 && k < P::A);
    double2 v[P::B], w[P::B];
    PB::load(z + q * P::LS, k, v);
#pragma unroll
    for (int r = 1; r < P::B; ++r) w[r] = tw[(r - 1) * P::A + k];
    PB::run(v, w);
    const long long ra = r0 + 2 * q;
    double* d = dst + ra * rps + k;
    if (ra < nrows) {
#pragma unroll
      for (int r = 0; r < P::B; ++r) d[r * P::A] = v[r].x;
    }
    if (ra + 1 < nrows) {
#pragma unroll
      for (int r = 0; r < P::B; ++r) d[rps + r * P::A] = v[r].y;
    }
  }
}

template <int L>
__global__ void __launch_bounds__(64, XLine<L>::MB) k_r2c2(FieldList in, long long rps, RowArr out, long long nrows,
                                                           int Kx, double scale, const double2* __restrict__ tw) {
  typedef XLine<L> P;
  typedef XPass<double2, L, P::A, 1, 0, false> PA;
  typedef XPass<double2, L, P::B, P::A, 0, false> PB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* z = (double2*)smem_raw;
  const double* src = (const double*)in.p[blockIdx.y];
  const long long r0 = (long long)blockIdx.x * (2 * P::NL);
  for (int i = threadIdx.x; i < P::NL * P::B; i += 64) {
    const int q = i / P::B, j = i - q * P::B;
    WFFT_ASSUME(j >= 0 && j < P::B);
    const long long ra = r0 + 2 * q;
    const bool oka = ra < nrows, okb = ra + 1 < nrows;
    const double* a = src + ra * rps + j;
    double2 v[P::A];
#pragma unroll
    for (int r = 0; r < P::A; ++r) {
      v[r].x = oka ? a[r * P::B] : 0.0;
      v[r].y = okb ? a[rps + r * P::B] : 0.0;
    }
    PA::run(v, nullptr);
    PA::store(z + q * P::LS, j, v);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < P::NL * P::A; i += 64) {
    const int q = i / P::A, k = i - q * P::A;
    WFFT_ASSUME(k >= 0 && k < P::A);
    double2 v[P::B], w[P::B];
    double2* line = z + q * P::LS;
    PB::load(line, k, v);
#pragma unroll
    for (int r = 1; r < P::B; ++r) w[r] = tw[(r - 1) * P::A + k];
    PB::run(v, w);
    PB::store(line, k, v);  // positions k + r RA, the ones it read
  }
  __syncthreads();
  const double sc = 0.5 * scale;
  double2* dst = (double2*)out.base + (long long)blockIdx.y * out.fs;
  for (int i = threadIdx.x; i < 2 * P::NL * Kx; i += 64) {
    const int rl = i / Kx, k = i - rl * Kx;
    if (r0 + rl >= nrows) break;
    const double2* line = z + (rl >> 1) * P::LS;
    const double2 zk = line[wsw<double2>(k)], zm = line[wsw<double2>(k ? L - k : 0)];
    dst[(r0 + rl) * out.rs + k] = (rl & 1) ? make_double2((zk.y + zm.y) * sc, (zm.x - zk.x) * sc)
                                           : make_double2((zk.x + zm.x) * sc, (zk.y - zm.y) * sc);
  }
}
