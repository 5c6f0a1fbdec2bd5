// Reference-layout (drop-in) streamwise and spanwise functions.
//
// Reference counterparts:
//   transform_3d_one (its 2D part) ........... source/transform.cu:95-319
//   computeLambVectorKernel .................. source/nonlinear.cu:307-428
#include "fftline.cuh"
#include "kernels.cuh"
#include "xline.cuh"
#include "zpass.cuh"
#include "zxline.cuh"
#include "zxpass.cuh"

// ---------------------------------------------------------------------------
// standalone streamwise C2R / R2C (drop-in transform_3d_one pieces)
// complex rows in [row][kx] (pitch rs) <-> real rows [row][x] (pitch rps)
// ---------------------------------------------------------------------------
template <typename C>
__global__ void k_x_c2r(RowArr in, T_of<C>* outr, long long rps, long long nrows, DnsGeom g,
                        FftTab<C> tab, int RB) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* z = (C*)smem_raw;  // RB/2 lines
  const int Px = g.Px;
  const int hx = g.Nx / 2;
  const long long r0 = (long long)blockIdx.x * RB;
  const int NP = RB / 2;
  for (int t = threadIdx.x; t < NP * Px; t += blockDim.x) {
    const int q = t / Px;
    const int n = t - q * Px;
    const long long ra = r0 + 2 * q, rb = ra + 1;
    C v = cmk<C>(0.0, 0.0);
    if (ra < nrows) {
      const C* a = prow<C>(in, 0, ra);
      // a last row without a neighbour is its own: the real part is its points
      const C* b = (rb < nrows) ? prow<C>(in, 0, rb) : a;
      v = pack_c2r<C>(a, b, n, Px, hx);
    }
    z[(size_t)q * Px + tab.drev[n]] = v;
  }
  fft_batch<C, true>(z, NP, Px, tab.plan, tab.tw);
  for (int t = threadIdx.x; t < RB * Px; t += blockDim.x) {
    const int rl = t / Px;
    const int j = t - rl * Px;
    const long long row = r0 + rl;
    if (row >= nrows) continue;
    const C v = z[(size_t)(rl / 2) * Px + j];
    outr[row * rps + j] = (rl & 1) ? v.y : v.x;
  }
}

template <typename C>
__global__ void k_x_r2c(const T_of<C>* inr, long long rps, RowArr out, long long nrows,
                        DnsGeom g, FftTab<C> tab, int RB, double scale) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef T_of<C> T;
  C* z = (C*)smem_raw;
  const int Px = g.Px;
  const long long r0 = (long long)blockIdx.x * RB;
  const int NP = RB / 2;
  for (int t = threadIdx.x; t < NP * Px; t += blockDim.x) {
    const int q = t / Px;
    const int j = t - q * Px;
    const long long ra = r0 + 2 * q, rb = ra + 1;
    C v = cmk<C>(0.0, 0.0);
    if (ra < nrows) v.x = inr[ra * rps + j];
    if (rb < nrows) v.y = inr[rb * rps + j];
    z[(size_t)q * Px + tab.drev[j]] = v;
  }
  fft_batch<C, false>(z, NP, Px, tab.plan, tab.tw);
  const int nk = Px / 2 + 1;  // the reference keeps all mx/2+1 bins
  const T sc = (T)(0.5 * scale);
  for (int t = threadIdx.x; t < RB * nk; t += blockDim.x) {
    const int rl = t / nk;
    const int k = t - rl * nk;
    const long long row = r0 + rl;
    if (row >= nrows) continue;
    const C v = unpack_r2c<C>(z + (size_t)(rl / 2) * Px, k, Px, (rl & 1) != 0);
    prow<C>(out, 0, row)[k] = v * sc;
  }
}

// pointwise Lamb vector on physical rows (drop-in computeLambVector):
// lambda may alias (u, v, w) as in the reference.
__global__ void k_lamb_rows(const double* u, const double* v, const double* w,
                            const double* ox, const double* oy, const double* oz,
                            double* lx, double* ly, double* lz, long long rps, int Px,
                            int Pz, long long nrows, const double* __restrict__ Uy, double Ro) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = idx / Px;
  const int j = (int)(idx - row * Px);
  if (row >= nrows) return;
  const long long o = row * rps + j;
  const double U = Uy[row / Pz];
  const double uu = u[o], vv = v[o], ww = w[o], a = ox[o], b = oy[o], c = oz[o];
  lx[o] = c * vv - b * ww - Ro * ww;
  ly[o] = a * ww - c * uu;
  lz[o] = b * uu - a * vv + Ro * (uu + U);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// Streamwise lines of nf fields.  Lengths with a plan take the two-butterfly
// form (us, before / after: three fields of 384 x 384 x 512 to points 1119 /
// 345, three of 192 x 192 x 256 to modes 163 / 59), other lengths one launch a
// field of the runtime-length form.
cudaError_t launch_x_c2r(RowArr in, FieldList out, int nf, long long rps, long long nrows, DnsGeom g,
                         FftTab<double2> tab, cudaStream_t st) {
  if (tab.zt && g.Nx / 2 == g.Px / 3) {
    const cudaError_t e = with_len_z(g.Px, [&](auto LL) -> cudaError_t {
      constexpr int L = decltype(LL)::value;
      typedef XLine<L> P;
      const size_t sm = (size_t)P::NL * P::LS * 16;
      k_c2r2<L><<<dim3((unsigned)((nrows + 2 * P::NL - 1) / (2 * P::NL)), nf), 64, sm, st>>>(in, out, rps, nrows, tab.zt);
      return cudaGetLastError();
    });
    if (e != cudaErrorNotSupported) return e;
  }
  const int RB = 4;
  const size_t sm = (size_t)(RB / 2) * g.Px * 16;
  cudaFuncSetAttribute(k_x_c2r<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  for (int f = 0; f < nf; ++f) {
    const RowArr rf{(double2*)in.base + (long long)f * in.fs, in.rs, 0};
    k_x_c2r<double2><<<(unsigned)((nrows + RB - 1) / RB), 256, sm, st>>>(rf, (double*)out.p[f], rps, nrows, g, tab, RB);
  }
  return cudaGetLastError();
}
cudaError_t launch_x_r2c(FieldList in, int nf, long long rps, RowArr out, long long nrows, DnsGeom g,
                         FftTab<double2> tab, double scale, cudaStream_t st) {
  if (tab.zt) {
    const cudaError_t e = with_len_z(g.Px, [&](auto LL) -> cudaError_t {
      constexpr int L = decltype(LL)::value;
      typedef XLine<L> P;
      const size_t sm = (size_t)P::NL * P::LS * 16;
      k_r2c2<L><<<dim3((unsigned)((nrows + 2 * P::NL - 1) / (2 * P::NL)), nf), 64, sm, st>>>(in, rps, out, nrows, g.Kx,
                                                                                          scale, tab.zt);
      return cudaGetLastError();
    });
    if (e != cudaErrorNotSupported) return e;
  }
  const int RB = 4;
  const size_t sm = (size_t)(RB / 2) * g.Px * 16;
  cudaFuncSetAttribute(k_x_r2c<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  for (int f = 0; f < nf; ++f) {
    const RowArr rf{(double2*)out.base + (long long)f * out.fs, out.rs, 0};
    k_x_r2c<double2><<<(unsigned)((nrows + RB - 1) / RB), 256, sm, st>>>((const double*)in.p[f], rps, rf, nrows, g, tab,
                                                                         RB, scale);
  }
  return cudaGetLastError();
}
// Spanwise passes of nf reference-layout fields (FP64), rows field by field
cudaError_t launch_zb_fields(PencilList in, RowArr out, int nf, DnsGeom g, FftTab<double2> tab, cudaStream_t st,
                             int variant) {
  if (variant == VAR_AUTO || variant == DNS_Z_WARP) {
    const cudaError_t e = launch_zb2<double2>(in, out, nf, g, tab, st, false);
    if (e != cudaErrorNotSupported) return e;
  }
  for (int f = 0; f < nf; ++f) {
    const cudaError_t e = launch_zb<double2>(PencilArr{in.f.p[f], in.ps, 0},
                                             RowArr{(double2*)out.base + (long long)f * out.fs, out.rs, 0}, 1, g, tab, st,
                                             nullptr, variant, false);
    if (e) return e;
  }
  return cudaSuccess;
}
cudaError_t launch_zf_fields(RowArr in, PencilList out, int nf, DnsGeom g, FftTab<double2> tab, cudaStream_t st,
                             int variant) {
  if (variant == VAR_AUTO || variant == DNS_Z_WARP) {
    const cudaError_t e = launch_zf2<double2>(in, out, nf, g, tab, st, false);
    if (e != cudaErrorNotSupported) return e;
  }
  for (int f = 0; f < nf; ++f) {
    const cudaError_t e = launch_zf<double2>(RowArr{(double2*)in.base + (long long)f * in.fs, in.rs, 0},
                                             PencilArr{out.f.p[f], out.ps, 0}, 1, g, tab, st, nullptr, variant, false);
    if (e) return e;
  }
  return cudaSuccess;
}
cudaError_t launch_lamb_rows(const double* const in6[6], double* const out3[3], long long rps,
                             long long nrows, DnsGeom g, const double* Uy, double Ro,
                             cudaStream_t st) {
  const long long n = nrows * g.Px;
  const int th = 256;
  k_lamb_rows<<<(unsigned)((n + th - 1) / th), th, 0, st>>>(
      in6[0], in6[1], in6[2], in6[3], in6[4], in6[5], out3[0], out3[1], out3[2], rps, g.Px, g.Pz,
      nrows, Uy, Ro);
  return cudaGetLastError();
}
