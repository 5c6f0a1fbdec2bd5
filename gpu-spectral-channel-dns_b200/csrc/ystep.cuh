// The time step's wall-normal passes: one pencil (kx, kz) per CTA.
//
// Reference counterparts:
//   getUVW + cheby_s2p ........... source/velocity.cu:22-170, source/transform.cu:416-748
//   cheby_p2s, rhsNonlinear ...... source/transform.cu:416-748, source/nonlinear.cu:130-242
//   worker s2p(No_Padding) ....... source/rhs.cpp:95-97
//   _get_linear_v / _omega_y / u0  source/linear.cpp:86-205
//   AB2 add ...................... source/rhs.cpp:205-215
//
// Lengths with a plan take the pruned DCT (ydct.cuh: k_y3d, k_y1d), others the
// block-wide FFT of the even extension (fft2.cuh, fft.cuh: k_y3, k_y1).
//
// ystep_f64.cu and ystep_f32.cu instantiate a precision each, and the drop-ins are
// modules of their own: a process loads the device code that it runs (with zxstep:
// first bootstrap of a process 4 ms in FP64, 7 mixed; 34 with everything in two
// modules, of which one took 21 ms to load and the other 28).
#pragma once
#include "fftline.cuh"
#include "kernels.cuh"
#include "mbar.cuh"
#include "ycoef.cuh"
#include "ydct.cuh"
#include "yline.cuh"
#include "ypass.cuh"

// ---------------------------------------------------------------------------
// Fused backward wall-normal pass (step start): getUVW from the FP64 state
// then the padded s2p of all six fields, written pencil-major for the
// spanwise pass.  Fields: u, v(span), w(wall), omega_x, omega_y, omega_z.
// ---------------------------------------------------------------------------
template <typename C, int LM>
__global__ void __launch_bounds__(256, 3) k_y3(const double2* __restrict__ V, const double2* __restrict__ O,
                     PencilArr out, DnsGeom g, PhysParams ph, FftTab<C> tab) {
  typedef FLine<C, LM> FL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Ny = g.Ny;
  const int M = tab.plan.L;  // 4 (Ny - 1)
  const int ls = FL::stride(M);
  Carve cv(smem_raw);
  double2* w = cv.take<double2>(Ny);
  double2* oz = cv.take<double2>(Ny);
  double2* Dw = cv.take<double2>(Ny);
  double2* u = cv.take<double2>(Ny);
  double2* v = cv.take<double2>(Ny);
  double2* Du = cv.take<double2>(Ny);
  double2* Dv = cv.take<double2>(Ny);
  double2* ox = cv.take<double2>(Ny);
  double2* oy = cv.take<double2>(Ny);
  C* lines = cv.take<C>((size_t)6 * ls);
  const long long p = blockIdx.x;
  int run, kx, kz;
  pencil_modes(g, p, run, kx, kz);
  const bool zero = (kx == 0 && kz == 0);
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = kmn_of(ia, ib);
  const double kmn1 = zero ? 0.0 : 1.0 / kmn;
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    w[n] = V[p * Ny + n];
    oz[n] = O[p * Ny + n];
  }
  __syncthreads();
  if (!zero && threadIdx.x < 32) ddz_warp(w, Dw, Ny);
  __syncthreads();
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    if (zero) {
      u[n] = w[n];
      v[n] = oz[n];
    } else {
      const double2 d = Dw[n], o = oz[n];
      u[n] = muli(d * (ia * kmn1)) - muli(o * (ib * kmn1));
      v[n] = muli(d * (ib * kmn1)) + muli(o * (ia * kmn1));
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  if (warp == 0) ddz_warp(v, Dv, Ny);
  if (warp == 1) ddz_warp(u, Du, Ny);
  __syncthreads();
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    const double2 wn = w[n];
    ox[n] = Dv[n] - muli(wn * ib);
    oy[n] = muli(wn * ia) - Du[n];
    if (zero) { w[n] = make_double2(0.0, 0.0); oz[n] = make_double2(0.0, 0.0); }
  }
  __syncthreads();
  const double2* src[6] = {u, v, w, ox, oy, oz};
  for (int t = threadIdx.x; t < 6 * M; t += blockDim.x) {
    const int f = t / M;
    const int n = t - f * M;
    lines[(size_t)f * ls + FL::in_pos(tab, n)] = from_d2<C>(ext_s2p_pad<C>(src[f], n, M, Ny));
  }
  FL::template fft<false>(lines, 6, ls, tab);
  const int Py = g.Py;
  for (int t = threadIdx.x; t < 6 * Py; t += blockDim.x) {
    const int f = t / Py;
    const int j = t - f * Py;
    pencil_ptr<C>(out, f, p)[j] = lines[(size_t)f * ls + FL::out_pos(j)];
  }
}

// Same pass with the six lines as pruned DCTs (ydct.cuh): two warps per
// pencil.  The FP64 state (by bulk copies), its derivatives and the exchange
// between the two passes share one region, the six fields' coefficients
// (halved for n > 0: the even extension) have their own.
//
// What bounds it: with whole 3-pass FFTs of the even extensions the pass moved
// each of 512 values of a line five times through shared memory and spent its
// issue slots on the redundant half; the two pruned passes move 0.56 of them
// once.  FP64 256 x 129 x 256 440 -> 301 us, 128 x 65 x 128 65 -> 50; mixed
// 144 x 55 x 72, a length on the block form before, 126 -> 21 (19 with the
// derivatives in FP32, which that length never had).
template <typename C, int M, int MB>
__global__ void __launch_bounds__(64, MB) k_y3d(const double2* __restrict__ V, const double2* __restrict__ O,
                                               PencilArr out, DnsGeom g, PhysParams ph, const C* __restrict__ dt,
                                               int* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef Dct<C, M, 6> D;
  constexpr int Ny = M / 4 + 1;  // the launcher checks g.Ny, g.Py against M
  typedef typename Y3Form<C, M>::E E;  // of the derivatives
  typedef T_of<E> S;
  constexpr int FS = (Ny + 1) & ~1;  // field stride
  C* fld = (C*)smem_raw;             // six fields
  unsigned char* rb = smem_raw + (size_t)6 * FS * sizeof(C);
  double2 *w = (double2*)rb, *oz = w + FS;
  E* eDw = (E*)(oz + FS);
  E *eD2w = eDw + FS, *eDoz = eD2w + FS, *ew = (E*)w, *eoz = (E*)oz;
  C* X = (C*)rb;
  const long long p = blockIdx.x;
  int run, kx, kz;
  pencil_modes(g, p, run, kx, kz);
  const bool zero = (kx == 0 && kz == 0);
  // the pencil's wavenumbers and 1 / k^2: the FP64 divisions once per CTA
  // (thread 0, under the copies), shared through shared memory
  __shared__ double pen[3];
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_expect_tx(&bar, (uint32_t)(2 * Ny * 16));
    bulk_g2s(w, V + p * Ny, (uint32_t)(Ny * 16), &bar);
    bulk_g2s(oz, O + p * Ny, (uint32_t)(Ny * 16), &bar);
    double a, b;
    wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, a, b);
    pen[0] = a;
    pen[1] = b;
    pen[2] = zero ? 0.0 : 1.0 / kmn_of(a, b);
  }
  __syncthreads();
  const double ia = pen[0], ib = pen[1], kmn1 = pen[2];
  if (!__syncthreads_and(mbar_wait_bounded(&bar, 0, ph.wait_limit, status))) {
    if (threadIdx.x == 0) {
      atomicOr(status, 1);
      mbar_wait_bounded(&bar, 0, DNS_WAIT_LIMIT, nullptr);  // let the copies land before leaving
    }
    return;
  }
  // derivatives: D w, D^2 w (warp 0) and D omega_z (warp 1); then, by
  // linearity, u = i(ia Dw - ib oz)/k^2, v = i(ib Dw + ia oz)/k^2 and their
  // derivatives from D^2 w, D oz (source/velocity.cu:90-170).  The mean
  // mode holds u0, w0 in (w, oz): u = w, v = oz, omega_x = D oz, omega_y = -D w.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (sizeof(E) == 8) {
    // to FP32 in place: element n of the FP32 copy lies below element n of
    // the FP64 vector, so the conversion runs in one pass per warp
    const double2* src = warp ? oz : w;
    E* dst = warp ? eoz : ew;
    for (int n0 = 0; n0 < Ny; n0 += 32) {
      const int n = n0 + lane;
      const double2 x = n < Ny ? src[n] : make_double2(0.0, 0.0);
      __syncwarp();
      if (n < Ny) dst[n] = make_float2((float)x.x, (float)x.y);
    }
    __syncwarp();
  }
  constexpr int CH = ddz_run(Ny);
  if (warp == 0) {
    ddz_fast<CH, E>(ew, eDw, Ny);
    __syncwarp();
    if (!zero) ddz_fast<CH, E>(eDw, eD2w, Ny);
  } else {
    ddz_fast<CH, E>(eoz, eDoz, Ny);
  }
  __syncthreads();
  const S sia = (S)(ia * kmn1), sib = (S)(ib * kmn1), fia = (S)ia, fib = (S)ib;
  for (int n = threadIdx.x; n < Ny; n += 64) {
    E wn = ew[n], on = eoz[n], u, v, ox, oy;
    const E d1 = eDw[n], dz = eDoz[n];
    if (zero) {
      u = wn;
      v = on;
      ox = dz;
      oy = cmk<E>(-d1.x, -d1.y);
      wn = on = cmk<E>(0.0, 0.0);  // w and omega_z vanish for the mean mode
    } else {
      const E d2 = eD2w[n];
      u = muli(d1 * sia) - muli(on * sib);
      v = muli(d1 * sib) + muli(on * sia);
      const E du = muli(d2 * sia) - muli(dz * sib);
      const E dv = muli(d2 * sib) + muli(dz * sia);
      ox = dv - muli(wn * fib);
      oy = muli(wn * fia) - du;
    }
    const S h = n ? (S)0.5 : (S)1.0;  // even extension: c_0, then c_n / 2
    fld[n] = from_e<C>(u * h);
    fld[FS + n] = from_e<C>(v * h);
    fld[2 * FS + n] = from_e<C>(wn * h);
    fld[3 * FS + n] = from_e<C>(ox * h);
    fld[4 * FS + n] = from_e<C>(oy * h);
    fld[5 * FS + n] = from_e<C>(on * h);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < D::IA; i += 64)
    D::template pass_a<Ny>(X, i, [&](int l, int n) { return fld[l * FS + n]; });
  __syncthreads();
  C* dst = pencil_ptr<C>(out, 0, p);
  for (int i = threadIdx.x; i < D::IB; i += 64)
    D::pass_b(X, dt, i, [&](int l, int k, C v) { dst[l * out.fs + k] = v; });
}

// ---------------------------------------------------------------------------
// Fused forward wall-normal pass: padded p2s of the three Lamb components,
// rhsNonlinear, then (unless boot) the right-hand sides of the banded
// wall-normal systems (wallsolve.h), all in Chebyshev coefficient space:
//
//   f = interpolant, at the Gauss-Lobatto points, of the reference's
//       collocation right-hand side (CN explicit operators, AB2 of the
//       nonlinear terms, v^n half of the tilting term; source/linear.cpp:
//       86-205, rhs.cpp:205-215).  Every term is a polynomial: derivatives
//       come from the coefficient recurrence, products with U(y), U'(y)
//       from multiplication by y, and the degrees above N fold back
//       (T_{N+j} = T_{N-j} at the Gauss-Lobatto points);
//   the equations do not use the walls (and, for v, the points next to
//       them): the interpolant with those values set to zero is f minus
//       f(y_m) times the cardinal polynomial of each such point y_m;
//   g = rows K .. K+n-1 of the K-fold Chebyshev integral (K = 4 for v, 2
//       for omega_y and the mean modes), the cardinal corrections taken from
//       precomputed integrated tables.
//
// The AB2 history is kept as Chebyshev coefficients of the nonlinear terms.
//   boot: only store the nonlinear terms as the AB2 history (the effect of
//         the reference's "extra previous step", source/main_loop.cpp:39-52).
// ---------------------------------------------------------------------------
namespace {
__device__ __forceinline__ double2 cget(const double2* X, int j, int N) {
  return (j >= 0 && j <= N) ? X[j] : make_double2(0.0, 0.0);
}
// coefficient j of y X (y T_0 = T_1, y T_i = (T_{i+1} + T_{i-1}) / 2)
__device__ __forceinline__ double2 ymul(const double2* X, int j, int N) {
  if (j < 0) return make_double2(0.0, 0.0);
  if (j == 0) return cget(X, 1, N) * 0.5;
  return (cget(X, j - 1, N) * (j == 1 ? 2.0 : 1.0) + cget(X, j + 1, N)) * 0.5;
}
__device__ __forceinline__ double2 y2mul(const double2* X, int j, int N) {
  if (j < 0) return make_double2(0.0, 0.0);
  if (j == 0) return ymul(X, 1, N) * 0.5;
  return (ymul(X, j - 1, N) * (j == 1 ? 2.0 : 1.0) + ymul(X, j + 1, N)) * 0.5;
}
// coefficient k of the Gauss-Lobatto interpolant of U(y) X(y)
__device__ __forceinline__ double2 umul_gl(const double2* X, int k, int N, const PhysParams& ph) {
  const bool quad = ph.U2 != 0.0;
  auto u = [&](int j) {
    double2 r = cget(X, j, N) * ph.U0 + ymul(X, j, N) * ph.U1;
    if (quad) r = r + y2mul(X, j, N) * ph.U2;
    return r;
  };
  double2 r = u(k);
  if (k == N - 1 || k == N - 2) r = r + u(2 * N - k);
  return r;
}
// ... of U'(y) X(y)
__device__ __forceinline__ double2 upmul_gl(const double2* X, int k, int N, const PhysParams& ph) {
  auto u = [&](int j) { return cget(X, j, N) * ph.U1 + ymul(X, j, N) * (2.0 * ph.U2); };
  double2 r = u(k);
  if (k == N - 1) r = r + u(N + 1);
  return r;
}
__device__ __forceinline__ double2 warp_sum(double2 v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, d);
    v.y += __shfl_down_sync(0xffffffffu, v.y, d);
  }
  return v;
}
}  // namespace

template <typename C, int LM>
__global__ void __launch_bounds__(256, 3) k_y1(PencilArr lam, const double2* __restrict__ V,
                                                const double2* __restrict__ O, double2* Nvp,
                                                double2* Nop, double2* gv, double2* go, RhsDims rd,
                                                RhsTabs tb, DnsGeom g, PhysParams ph,
                                                FftTab<C> tabP, int boot) {
  typedef FLine<C, LM> FP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Ny = g.Ny;
  const int Py = g.Py;
  const int N = Ny - 1;
  const int M = tabP.plan.L;  // 2 (Py - 1)
  const int lsP = FP::stride(M);
  const int LB = Ny + 8;
  Carve cv(smem_raw);
  double2* lc = cv.take<double2>((size_t)3 * Ny);  // lambda coefficients, then fv, fo
  double2* D1 = cv.take<double2>((size_t)2 * Ny);  // D lambda_x, D lambda_y
  double2* Vc = cv.take<double2>(Ny);
  double2* Oc = cv.take<double2>(Ny);
  double2* nvc = cv.take<double2>(Ny);
  double2* noc = cv.take<double2>(Ny);
  double2* DV = cv.take<double2>(Ny);
  double2* D2V = cv.take<double2>(Ny);
  double2* D3V = cv.take<double2>(Ny);
  double2* D4V = cv.take<double2>(Ny);
  double2* DO = cv.take<double2>(Ny);
  double2* D2O = cv.take<double2>(Ny);
  double2* red = cv.take<double2>(8);  // values of fv, fo at the unused points
  const size_t bytesP = (size_t)3 * lsP * sizeof(C), bytesI = (size_t)4 * LB * 16;
  unsigned char* region = cv.take<unsigned char>(bytesP > bytesI ? bytesP : bytesI);
  C* linesP = (C*)region;

  const long long p = blockIdx.x;
  int run, kx, kz;
  pencil_modes(g, p, run, kx, kz);
  const bool zero = (kx == 0 && kz == 0);
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = kmn_of(ia, ib);

  // 1. Lamb pencils as even extensions (DCT-I of Py points); state, history
  for (int t = threadIdx.x; t < 3 * M; t += blockDim.x) {
    const int f = t / M;
    const int n = t - f * M;
    const C* src = pencil_ptr<C>(lam, f, p);
    linesP[(size_t)f * lsP + FP::in_pos(tabP, n)] = (n < Py) ? src[n] : src[M - n];
  }
  if (!boot)
    for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
      Vc[n] = V[p * Ny + n];
      Oc[n] = O[p * Ny + n];
      nvc[n] = Nvp[p * Ny + n];
      noc[n] = Nop[p * Ny + n];
    }
  FP::template fft<false>(linesP, 3, lsP, tabP);
  const double sc = 1.0 / (Py - 1);
  for (int t = threadIdx.x; t < 3 * Ny; t += blockDim.x) {
    const int f = t / Ny;
    const int k = t - f * Ny;
    double2 c = to_d2(linesP[(size_t)f * lsP + FP::out_pos(k)]) * sc;
    if (k == 0) c = c * 0.5;
    lc[t] = c;
  }
  __syncthreads();
  // 2. derivatives (independent chains on separate warps)
  const int warp = threadIdx.x >> 5;
  if (warp == 0) ddz_warp(lc, D1, Ny);
  if (warp == 1) ddz_warp(lc + Ny, D1 + Ny, Ny);
  if (!boot) {
    if (warp == 2) {
      ddz_warp(Vc, DV, Ny);
      __syncwarp();
      ddz_warp(DV, D2V, Ny);
      __syncwarp();
      ddz_warp(D2V, D3V, Ny);
      __syncwarp();
      ddz_warp(D3V, D4V, Ny);
    }
    if (warp == 3) {
      ddz_warp(Oc, DO, Ny);
      __syncwarp();
      ddz_warp(DO, D2O, Ny);
    }
  }
  __syncthreads();
  // 3. nonlinear terms (coefficients) -> history; interpolated right-hand sides
  const double dt = run_dt(ph, run), Re = run_Re(ph, run), gam = ia * dt * 0.5;
  const double kap = -0.5 * ib * dt;  // tilting weight (source/linear.cpp:147-151)
  double2* fv = lc;
  double2* fo = lc + Ny;
  for (int k = threadIdx.x; k < Ny; k += blockDim.x) {
    double2 hv, ho;
    if (zero) {
      hv = lc[k];
      ho = lc[Ny + k];
    } else {
      hv = lc[2 * Ny + k] * kmn + muli(D1[k] * ia) + muli(D1[Ny + k] * ib);
      ho = muli(lc[Ny + k] * ia) - muli(lc[k] * ib);
    }
    Nvp[p * Ny + k] = hv;
    Nop[p * Ny + k] = ho;
    if (boot) continue;
    double2 a, b;
    if (zero) {
      // _get_linear_u0 / _w0
      a = Vc[k] + D2V[k] * (dt * 0.5 / Re) - (hv * 1.5 - nvc[k] * 0.5) * dt;
      b = Oc[k] + D2O[k] * (dt * 0.5 / Re) - (ho * 1.5 - noc[k] * 0.5) * dt;
    } else {
      const double2 re = D4V[k] * (dt * 0.5 / Re) + D2V[k] * (1 - kmn * dt / Re)
                         - Vc[k] * (kmn * (1 - kmn * dt * 0.5 / Re));
      const double2 im = umul_gl(D2V, k, N, ph) * (-gam) + umul_gl(Vc, k, N, ph) * (kmn * gam)
                         + Vc[k] * (gam * 2.0 * ph.U2);
      a = re + muli(im) + (hv * 1.5 - nvc[k] * 0.5) * dt;
      const double2 ro = D2O[k] * (0.5 / Re * dt) + Oc[k] * (1 - kmn * dt * 0.5 / Re);
      b = ro + muli(umul_gl(Oc, k, N, ph) * (-gam)) + (ho * 1.5 - noc[k] * 0.5) * dt
          + muli(upmul_gl(Vc, k, N, ph) * kap);
    }
    fv[k] = a;
    fo[k] = b;
  }
  if (boot) return;
  __syncthreads();
  // 4. values at the points the equations leave out; integration buffers
  double2* av = (double2*)region;
  double2* bv = av + LB;
  double2* ao = bv + LB;
  double2* bo = ao + LB;
  const int lane = threadIdx.x & 31;
  if (warp < 2) {
    const double2* f = warp ? fo : fv;
    double2 s0 = make_double2(0.0, 0.0), sN = s0, s1 = s0, sN1 = s0;
    for (int k = lane; k < Ny; k += 32) {
      const double2 v = f[k];
      const double cs = __ldg(tb.cosk + k);
      const double sg = (k & 1) ? -1.0 : 1.0;
      s0 = s0 + v;
      sN = sN + v * sg;
      s1 = s1 + v * cs;
      sN1 = sN1 + v * (sg * cs);
    }
    s0 = warp_sum(s0);
    sN = warp_sum(sN);
    s1 = warp_sum(s1);
    sN1 = warp_sum(sN1);
    if (lane == 0) {
      red[4 * warp + 0] = s0;   // y = 1
      red[4 * warp + 1] = s1;   // y_1
      red[4 * warp + 2] = sN1;  // y_{N-1}
      red[4 * warp + 3] = sN;   // y = -1
    }
  } else {
    for (int t = threadIdx.x - 64; t < 2 * LB; t += blockDim.x - 64) {
      const int f = t / LB;
      const int k = t - f * LB;
      (f ? ao : av)[k] = (k <= N) ? (f ? fo : fv)[k] : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  // 5. Chebyshev integration (B x)_k = (c_{k-1} x_{k-1} - x_{k+1}) / (2k), (B x)_0 = 0
  const int Kv = zero ? 2 : 4;
  for (int it = 0; it < Kv; ++it) {
    const int nf = (it < 2) ? 2 : 1;
    for (int t = threadIdx.x; t < nf * LB; t += blockDim.x) {
      const int f = t / LB;
      const int k = t - f * LB;
      const double2* x = f ? ao : av;
      double2* y = f ? bo : bv;
      double2 r = make_double2(0.0, 0.0);
      if (k >= 1) {
        const double2 xm = x[k - 1] * (k == 1 ? 2.0 : 1.0);
        const double2 xp = (k + 1 < LB) ? x[k + 1] : make_double2(0.0, 0.0);
        r = (xm - xp) * (1.0 / (2.0 * k));
      }
      y[k] = r;
    }
    __syncthreads();
    double2* tmp = av; av = bv; bv = tmp;
    if (it < 2) { tmp = ao; ao = bo; bo = tmp; }
  }
  // 6. rows K .. K+n-1 minus the integrated cardinal corrections
  for (int r = threadIdx.x; r < rd.nv; r += blockDim.x) {
    double2 v = (Kv + r < LB) ? av[Kv + r] : make_double2(0.0, 0.0);
    if (zero) {
      v = v - red[0] * __ldg(tb.bkco + r) - red[3] * __ldg(tb.bkco + rd.no + r);
    } else {
#pragma unroll
      for (int m = 0; m < 4; ++m) v = v - red[m] * __ldg(tb.bkcv + (size_t)m * rd.nv + r);
    }
    gv[p * rd.gp + r] = v;
  }
  for (int r = threadIdx.x; r < rd.no; r += blockDim.x) {
    double2 v = (2 + r < LB) ? ao[2 + r] : make_double2(0.0, 0.0);
    v = v - red[4] * __ldg(tb.bkco + r) - red[7] * __ldg(tb.bkco + rd.no + r);
    go[p * rd.gp + r] = v;
  }
}

// Same pass with the three lines as pruned DCTs (ydct.cuh) on warps 0 and 1
// (which then differentiate lambda_x and lambda_y), the parts of the
// right-hand sides that need the state only on warps 2 and 3 meanwhile.
//
// The integrated right-hand side is formed without D^2 v and D^4 v.  From row
// 4 on, B^4 D^4 v = v and B^4 D^2 v = B^2 v, and
//   U D^2 v = D^2 (U v) - 2 D (U' v) + U'' v
// (degree <= N: its interpolant is itself), so with h = dt / (2 Re), gam =
// alpha dt / 2, P = U v (degree <= N + 2) and Pf its interpolant
//   g = h v + B^2 [(1 - 2 k^2 h) v - i gam P] + B^3 [2 i gam U' v]
//       + B^4 [-k^2 (1 - k^2 h) v + i gam k^2 Pf + dt (1.5 N - 0.5 N_p)]
// (the two U'' terms cancel); for omega_y and the mean modes, from row 2 on,
//   g = h o + B^2 [(1 - k^2 h) o - i gam (U o)f + i kap (U' v)f + dt (...)].
// The values at the left-out points take the derivatives of T_k there; H_v
// takes one derivative, of alpha lambda_x + beta lambda_y.
//
// What bounds it: issue slots (7055 warp instructions a pencil at M = 512
// before, a fifth of them FP64), so vectors carry zero guards instead of
// bounds checks, and the sums over k are halved between lanes at every
// step.  4530 instructions; 256 x 129 x 256 mixed 383 -> 278 us, FP64 497 ->
// 432; 128 x 65 x 128 FP64 107 -> 63; twelve 64 x 49 x 64 mixed 184 -> 114;
// 144 x 55 x 72 mixed, a length on the block form before, 160 -> 33.
template <typename C, int M, int MB>
__global__ void __launch_bounds__(128, MB) k_y1d(PencilArr lam, const double2* __restrict__ V,
                                            const double2* __restrict__ O, double2* Nvp,
                                            double2* Nop, double2* gv, double2* go, RhsDims rd,
                                            RhsTabs tb, DnsGeom g, PhysParams ph,
                                            const C* __restrict__ dct, int boot, int* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef Dct<C, M, 3> D;
  constexpr int Ny = M / 4 + 1;  // the launcher checks g.Ny, g.Py against M
  constexpr int Py = M / 2 + 1;
  constexpr int N = Ny - 1;
  constexpr int PS = (Py + 1) & ~1;      // staged Lamb pencil
  constexpr int GU = 12, VL = Ny + GU;   // zero guards above N (two more below 0 for v and omega)
  Carve cv(smem_raw);
  double2* Vc = cv.take<double2>(VL + 2) + 2;
  double2* Oc = cv.take<double2>(VL + 2) + 2;
  double2* nvc = cv.take<double2>(Ny);
  double2* noc = cv.take<double2>(Ny);
  double2* S2 = cv.take<double2>(VL);  // under B^2
  double2* S4 = cv.take<double2>(VL);  // under B^4 (mean modes: B^2)
  double2* T2 = cv.take<double2>(VL);  // omega: under B^2
  double2* red = cv.take<double2>(6);  // right-hand sides at the left-out points: v 1, y_1, -y_1, -1; omega 1, -1
  double* accA = cv.take<double>(2 * 2 * 10);  // [warp - 2][parity][value]: derivatives of the state there
  double* accB = cv.take<double>(4 * 2 * 6);   // [warp][parity][value]: the rest there
  // the staged Lamb pencils, then the coefficients of lambda; the exchange of
  // the transform, then alpha lambda_x + beta lambda_y and its derivative
  constexpr size_t LB = sizeof(C) * 3 * PS, LC = (size_t)16 * 3 * Ny, XB = sizeof(C) * D::XN, XD = (size_t)16 * 2 * Ny;
  C* stg = (C*)cv.take<unsigned char>(LB > LC ? LB : LC);
  C* X = (C*)cv.take<unsigned char>(XB > XD ? XB : XD);
  double2 *lx = (double2*)stg, *ly = lx + Ny, *lz = ly + Ny;
  double2 *q = (double2*)X, *Dq = q + Ny;

  const long long p = blockIdx.x;
  int run, kx, kz;
  pencil_modes(g, p, run, kx, kz);
  const bool zero = (kx == 0 && kz == 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the pencil's wavenumbers, k^2, dt and dt / (2 Re): the FP64 divisions
  // once per CTA (thread 0, under the copies), shared through shared memory
  __shared__ double pen[5];

  // 1. bulk copies on one barrier: the three Lamb pencils, state, history
  const uint32_t lamb = (uint32_t)(PS * sizeof(C));
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_expect_tx(&bar, 3 * lamb + (boot ? 0u : (uint32_t)(4 * Ny * 16)));
    for (int f = 0; f < 3; ++f) bulk_g2s(stg + (size_t)f * PS, pencil_ptr<C>(lam, f, p), lamb, &bar);
    if (!boot) {
      bulk_g2s(Vc, V + p * Ny, (uint32_t)(Ny * 16), &bar);
      bulk_g2s(Oc, O + p * Ny, (uint32_t)(Ny * 16), &bar);
      bulk_g2s(nvc, Nvp + p * Ny, (uint32_t)(Ny * 16), &bar);
      bulk_g2s(noc, Nop + p * Ny, (uint32_t)(Ny * 16), &bar);
    }
    double a, b;
    wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, a, b);
    const double dt = run_dt(ph, run), Re = run_Re(ph, run);
    pen[0] = a;
    pen[1] = b;
    pen[2] = kmn_of(a, b);
    pen[3] = dt;
    pen[4] = dt * 0.5 / Re;
  } else if (threadIdx.x >= 64 && threadIdx.x < 64 + GU + 2) {
    const int i = threadIdx.x - 64 - 2;  // -2 .. GU - 1
    const double2 z2 = make_double2(0.0, 0.0);
    Vc[i < 0 ? i : Ny + i] = z2;
    Oc[i < 0 ? i : Ny + i] = z2;
    if (i >= 0) S4[Ny + i] = T2[Ny + i] = S2[Ny + i] = z2;  // (S2 N + 1, N + 2 written below)
  }
  __syncthreads();
  const double ia = pen[0], ib = pen[1], kmn = pen[2];
  if (!__syncthreads_and(mbar_wait_bounded(&bar, 0, ph.wait_limit, status))) {
    if (threadIdx.x == 0) {
      atomicOr(status, 1);
      mbar_wait_bounded(&bar, 0, DNS_WAIT_LIMIT, nullptr);  // let the copies land before leaving
    }
    return;
  }
  const double dt = pen[3], h = pen[4], gam = zero ? 0.0 : ia * dt * 0.5;
  // 2. warps 0, 1: transforms, derivative; warps 2, 3: the state's part of
  //    the right-hand sides, its derivatives at the left-out points
  if (warp < 2) {
    auto pair = []() { asm volatile("bar.sync 1, 64;" ::: "memory"); };
    for (int i = threadIdx.x; i < D::IA; i += 64)
      D::template pass_a<0>(X, i, [&](int l, int n) { return stg[l * PS + n]; });
    pair();
    for (int i = threadIdx.x; i < D::IB; i += 64)
      D::pass_b(X, dct, i, [&](int l, int k, C v) {
        if (k < Ny) lx[l * Ny + k] = to_d2(v) * (k ? 1.0 / (Py - 1) : 0.5 / (Py - 1));
      });
    pair();
    for (int k = threadIdx.x; k < Ny; k += 64) q[k] = lx[k] * ia + ly[k] * ib;
    pair();
    if (warp == 0) ddz_fast<ddz_run(Ny)>(q, Dq, Ny);
  } else if (!boot) {
    const double c2v = 1 - 2.0 * kmn * h, c0v = kmn * (1 - kmn * h), c0o = 1 - kmn * h;
    const double kap = -0.5 * ib * dt;  // tilting weight (source/linear.cpp:147-151)
    double acc[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) acc[i] = 0.0;
    for (int k = threadIdx.x - 64; k < Ny + 2; k += 64) {
      const double2 v = Vc[k];
      double2 P, Pf;
      u_times(Vc, k, N, ph, P, Pf);
      S2[k] = make_double2(v.x * c2v + P.y * gam, v.y * c2v - P.x * gam);
      if (k < Ny) {
        const double kg = kmn * gam;
        S4[k] = zero ? v : make_double2(-(v.x * c0v + Pf.y * kg), Pf.x * kg - v.y * c0v);
        const double2 o = Oc[k];
        double2 Q, Qf;
        u_times(Oc, k, N, ph, Q, Qf);
        const double2 im = up_times(Vc, k, N, ph) * kap - Qf * gam;
        T2[k] = zero ? o : make_double2(o.x * c0o - im.y, o.y * c0o + im.x);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const double w = __ldg(tb.tw + t * Ny + k);
          acc[2 * t] += v.x * w;
          acc[2 * t + 1] += v.y * w;
        }
        const double w = __ldg(tb.tw + k);
        acc[8] += o.x * w;
        acc[9] += o.y * w;
      }
    }
    const double sum = ParitySums<10>::run(acc, lane);
    const int idx = ParitySums<10>::slot(lane);
    if (idx < 10) accA[((warp - 2) * 2 + (lane & 1)) * 10 + idx] = sum;
  }
  __syncthreads();
  // 3. nonlinear terms (coefficients) -> history, and into the right-hand
  //    sides; sums of these for the left-out points
  const double dtn = zero ? -dt : dt;
  double acc[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) acc[i] = 0.0;
  for (int k = threadIdx.x; k < Ny; k += 128) {
    const double2 x = lx[k], y = ly[k];
    double2 hv = x, ho = y;
    if (!zero) {
      const double2 z = lz[k], d = Dq[k];
      hv = make_double2(z.x * kmn - d.y, z.y * kmn + d.x);
      ho = make_double2(x.y * ib - y.y * ia, y.x * ia - x.x * ib);
    }
    Nvp[p * Ny + k] = hv;
    Nop[p * Ny + k] = ho;
    if (boot) continue;
    const double2 s4 = S4[k] + (hv * 1.5 - nvc[k] * 0.5) * dtn;
    const double2 t2 = T2[k] + (ho * 1.5 - noc[k] * 0.5) * dtn;
    S4[k] = s4;
    T2[k] = t2;
    double2 f = s4;
    if (ph.U2 != 0.0) f = f + muli(Vc[k]) * (2.0 * gam * ph.U2);
    const double c = __ldg(tb.cosk + k);
    acc[0] += f.x;
    acc[1] += f.y;
    acc[2] += f.x * c;
    acc[3] += f.y * c;
    acc[4] += t2.x;
    acc[5] += t2.y;
  }
  if (boot) return;
  {
    const double sum = ParitySums<6>::run(acc, lane);
    const int idx = ParitySums<6>::slot(lane);
    if (idx < 6) accB[(warp * 2 + (lane & 1)) * 6 + idx] = sum;
  }
  __syncthreads();
  // 4. right-hand sides at the points the equations leave out (six threads);
  //    the mean modes are two systems of the omega kind
  if (threadIdx.x >= 96 && threadIdx.x < 102) {
    const int i = threadIdx.x - 96, at = i == 1 || i == 2;  // at +-y_1
    const double sg = (i == 2 || i == 3 || i == 5) ? -1.0 : 1.0;
    auto sumA = [&](int v) {
      const double* a = accA + v;
      return make_double2(a[0] + a[20] + (a[10] + a[30]) * sg, a[1] + a[21] + (a[11] + a[31]) * sg);
    };
    const double* a = accB + (i >= 4 ? 4 : 2 * at);
    double2 f = make_double2(0.0, 0.0);
#pragma unroll
    for (int w = 0; w < 4; ++w) f = f + make_double2(a[12 * w] + a[12 * w + 6] * sg, a[12 * w + 1] + a[12 * w + 7] * sg);
    if (i >= 4 || zero) {
      f = f + sumA(i >= 4 ? 8 : 0) * h;
    } else {
      const double y = (at ? __ldg(tb.cosk + 1) : 1.0) * sg;
      const double2 d2 = sumA(4 * at), d4 = sumA(4 * at + 2);
      f = f + d4 * h + d2 * (1 - 2.0 * kmn * h) - muli(d2) * (gam * (ph.U0 + (ph.U1 + ph.U2 * y) * y));
    }
    red[i] = f;
  }
  //    and the integrals by their banded stencils (all threads)
  constexpr int RPT = (Ny + 2 + 127) / 128;  // rows per thread (n <= Ny + 2, 128 threads)
  const int n2 = rd.nv + 2;
  double2 iv[RPT], io[RPT];
#pragma unroll
  for (int t = 0; t < RPT; ++t) {
    const int r = threadIdx.x + t * 128;
    iv[t] = io[t] = make_double2(0.0, 0.0);
    if (r < rd.nv) {
      const double* b2 = tb.b2 + r;
      double w[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) w[d] = __ldg(b2 + d * n2);
      io[t] = Oc[r + 2] * h;
#pragma unroll
      for (int d = 0; d < 3; ++d) io[t] = io[t] + T2[r + 2 * d] * w[d];
      if (zero) {
        iv[t] = Vc[r + 2] * h;
#pragma unroll
        for (int d = 0; d < 3; ++d) iv[t] = iv[t] + S4[r + 2 * d] * w[d];
      } else {
        iv[t] = Vc[r + 4] * h;
        const double* b4 = tb.b4 + r;
#pragma unroll
        for (int d = 0; d < 5; ++d) iv[t] = iv[t] + S4[r + 2 * d] * __ldg(b4 + d * rd.nv);
#pragma unroll
        for (int d = 0; d < 3; ++d) iv[t] = iv[t] + S2[r + 2 + 2 * d] * __ldg(b2 + d * n2 + 2);
        if (ph.U1 != 0.0 || ph.U2 != 0.0) {
          double2 s3 = make_double2(0.0, 0.0);
          const double* b3 = tb.b3 + r;
#pragma unroll
          for (int d = 0; d < 4; ++d) {
            const int k = r + 1 + 2 * d;
            double2 x = Vc[k] * ph.U1;
            if (ph.U2 != 0.0) x = x + (Vc[k - 1] * (k == 1 ? 2.0 : 1.0) + Vc[k + 1]) * ph.U2;
            s3 = s3 + x * __ldg(b3 + d * rd.nv);
          }
          iv[t] = iv[t] + muli(s3) * (2.0 * gam);
        }
      }
    }
  }
  __syncthreads();
  // 5. minus the integrated cardinal corrections, out
#pragma unroll
  for (int t = 0; t < RPT; ++t) {
    const int r = threadIdx.x + t * 128;
    if (r < rd.nv) {  // as many rows of omega
      const double c0 = __ldg(tb.bkco + r), cN = __ldg(tb.bkco + rd.no + r);
      double2 v = iv[t];
      if (zero) {
        v = v - red[0] * c0 - red[3] * cN;
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) v = v - red[m] * __ldg(tb.bkcv + m * rd.nv + r);
      }
      gv[p * rd.gp + r] = v;
      go[p * rd.gp + r] = io[t] - red[4] * c0 - red[5] * cN;
    }
  }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
inline size_t y3_smem(int Ny, int ls, size_t csz) {
  auto a = [](size_t b) { return (b + 15) & ~(size_t)15; };
  return 9 * a((size_t)Ny * 16) + a((size_t)6 * ls * csz);
}
inline size_t y1_smem(int Ny, int lsP, size_t csz) {
  auto a = [](size_t b) { return (b + 15) & ~(size_t)15; };
  size_t s = a((size_t)3 * Ny * 16) + a((size_t)2 * Ny * 16) + 10 * a((size_t)Ny * 16) + a(8 * 16);
  size_t bp = (size_t)3 * lsP * csz, bi = (size_t)4 * (Ny + 8) * 16;
  return s + a(bp > bi ? bp : bi);
}

template <typename C>
cudaError_t launch_y3(const double2* V, const double2* O, PencilArr out, DnsGeom g,
                      PhysParams ph, FftTab<C> tab, int* status, cudaStream_t st, int variant, bool probe) {
  const bool any = variant == VAR_AUTO;
  // the warp form stages its inputs by bulk copies (16-byte aligned
  // sources) and takes Ny = M/4 + 1, Py = M/2 + 1 as compile-time constants
  if ((any || variant == DNS_Y3_FFT) && aligned16(V) && aligned16(O) && tab.dt && g.Ny == tab.plan.L / 4 + 1 &&
      g.Py == tab.plan.L / 2 + 1) {
    const cudaError_t e = with_len_d(tab.plan.L, [&](auto MM) -> cudaError_t {
      constexpr int M = decltype(MM)::value;
      typedef Dct<C, M, 6> D;
      if (probe) return cudaSuccess;
      constexpr int FS = (M / 4 + 2) & ~1;
      constexpr size_t es = sizeof(typename Y3Form<C, M>::E), vec = (size_t)FS * (2 * 16 + 3 * es), ex = D::XN * sizeof(C);
      const size_t sm = (size_t)6 * FS * sizeof(C) + (vec > ex ? vec : ex);
      constexpr int MB = sizeof(C) == 8 ? (D::RA > 18 ? 8 : 12) : (D::RA > 24 ? 4 : (D::RA > 18 ? 6 : 8));
      auto k = k_y3d<C, M, MB>;
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      k<<<(unsigned)g.H, 64, sm, st>>>(V, O, out, g, ph, tab.dt, status);
      return cudaGetLastError();
    });
    if (e != cudaErrorNotSupported) return e;
  }
  if (!any && variant != DNS_Y3_BLOCK) return cudaErrorNotSupported;
  if (probe) return cudaSuccess;
  return with_len_m(tab.plan.L, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    const size_t sm = y3_smem(g.Ny, FLine<C, L>::stride(tab.plan.L), sizeof(C));
    cudaFuncSetAttribute(k_y3<C, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_y3<C, L><<<(unsigned)g.H, 256, sm, st>>>(V, O, out, g, ph, tab);
    return cudaGetLastError();
  });
}

// CTAs per SM of k_y1d, by the first radix (its registers). The kernel waits at
// barriers between short phases, so one more resident CTA is worth a few spilled
// words: with 5 | 6 | 8 (FP32) and 3 | 4 | 4 (FP64) CTAs 84x33x84 took 31.0 us
// (now 25.4), 128x65x128 74.6 (63.4), mixed 256x129x256 300 (277), FP64
// 256x129x256 442 (432); one CTA more again, 10 in FP32, 5 % slower.
template <typename C, int M> constexpr int y1_ctas() {
  constexpr int RA = DPlan<M>::A;
  return sizeof(C) == 8 ? (RA > 24 ? 7 : (RA > 18 ? 8 : 9)) : (RA > 24 ? 4 : (RA > 16 ? 5 : 7));
}
template <typename C>
cudaError_t launch_y1(PencilArr lam, const double2* V, const double2* O, double2* Nvp,
                      double2* Nop, double2* gv, double2* go, RhsDims rd, RhsTabs tb, DnsGeom g,
                      PhysParams ph, FftTab<C> tabP, int boot, int* status, cudaStream_t st, int variant,
                      bool probe) {
  const bool any = variant == VAR_AUTO;
  // the warp form stages its inputs by bulk copies (16-byte aligned pencils
  // with room for Py rounded up to even) and takes Ny = M/4 + 1,
  // Py = M/2 + 1 as compile-time constants
  const bool bulk_ok = aligned16(lam.base) && (lam.ps * sizeof(C)) % 16 == 0 &&
                       (lam.fs * sizeof(C)) % 16 == 0 && lam.ps >= ((g.Py + 1) & ~1) && aligned16(V) &&
                       aligned16(O) && aligned16(Nvp) && aligned16(Nop) && tabP.dt &&
                       g.Ny == tabP.plan.L / 4 + 1 && g.Py == tabP.plan.L / 2 + 1;
  if ((any || variant == DNS_Y1_WARP) && bulk_ok) {
    const cudaError_t e = with_len_d(tabP.plan.L, [&](auto MM) -> cudaError_t {
      constexpr int M = decltype(MM)::value;
      typedef Dct<C, M, 3> D;
      if (probe) return cudaSuccess;
      auto a = [](size_t b) { return (b + 15) & ~(size_t)15; };
      const size_t lb = sizeof(C) * 3 * ((g.Py + 1) & ~1), lc = (size_t)48 * g.Ny, xb = sizeof(C) * D::XN,
                   xd = (size_t)32 * g.Ny;
      // vectors with their guards, sums, staged pencils, exchange (as carved)
      const size_t sm = (size_t)(7 * g.Ny + 5 * 12 + 4 + 6) * 16 + (40 + 48) * 8 + a(lb > lc ? lb : lc) + a(xb > xd ? xb : xd);
      auto k = k_y1d<C, M, y1_ctas<C, M>()>;
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      k<<<(unsigned)g.H, 128, sm, st>>>(lam, V, O, Nvp, Nop, gv, go, rd, tb, g, ph, tabP.dt, boot, status);
      return cudaGetLastError();
    });
    if (e != cudaErrorNotSupported) return e;
  }
  if (!any && variant != DNS_Y1_BLOCK) return cudaErrorNotSupported;
  if (probe) return cudaSuccess;
  return with_len_m(tabP.plan.L, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    const size_t sm = y1_smem(g.Ny, FLine<C, L>::stride(tabP.plan.L), sizeof(C));
    cudaFuncSetAttribute(k_y1<C, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_y1<C, L><<<(unsigned)g.H, 256, sm, st>>>(lam, V, O, Nvp, Nop, gv, go, rd, tb, g, ph, tabP, boot);
    return cudaGetLastError();
  });
}
