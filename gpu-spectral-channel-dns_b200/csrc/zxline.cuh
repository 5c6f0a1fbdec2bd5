// Device helpers of the spanwise and streamwise kernels (zxpass.cu, zxstep.cuh).
#pragma once
#include "kernels.cuh"

namespace {
template <typename C>
__device__ __forceinline__ C* prow(const RowArr& a, int f, long long row) {
  return (C*)a.base + (long long)f * a.fs + row * a.rs;
}
template <typename C>
__device__ __forceinline__ C* ppen(const PencilArr& a, int f, long long p) {
  return (C*)a.base + (long long)f * a.fs + p * a.ps;
}
}  // namespace

namespace {
// Hermitian half-spectra a, b (bins 0..Kx-1, Nyquist and padding zero) packed
// as Z = A + iB over the full length Px, so that IFFT(Z) = a(x) + i b(x).
// The imaginary parts of the DC bins are dropped (C2R convention).
template <typename C>
__device__ __forceinline__ C pack_c2r(const C* a, const C* b, int n, int Px, int hx) {
  if (n == 0) return cmk<C>((double)a[0].x, (double)b[0].x);
  if (n < hx) {
    const C av = a[n], bv = b[n];
    C z; z.x = av.x - bv.y; z.y = av.y + bv.x; return z;
  }
  if (n > Px - hx) {
    const int k = Px - n;
    const C av = a[k], bv = b[k];
    C z; z.x = av.x + bv.y; z.y = bv.x - av.y; return z;  // conj(a) + i conj(b)
  }
  return cmk<C>(0.0, 0.0);
}
// unpack the spectra of the real and imaginary parts of a complex signal
template <typename C>
__device__ __forceinline__ C unpack_r2c(const C* Z, int k, int Px, bool imag_part) {
  const C zk = Z[k];
  const C zm = Z[(Px - k) % Px];
  C r;
  if (!imag_part) { r.x = (zk.x + zm.x); r.y = (zk.y - zm.y); }   // Zk + conj(Zm)
  else { r.x = (zk.y + zm.y); r.y = (zm.x - zk.x); }              // -i (Zk - conj(Zm))
  return r;
}
}  // namespace
