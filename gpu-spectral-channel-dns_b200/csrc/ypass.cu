// Reference-layout (drop-in) wall-normal functions: one or a few pencils per CTA.
//
// Reference counterparts:
//   cheby_s2p / cheby_p2s ........ source/transform.cu:416-748
//   getUVW ....................... source/velocity.cu:22-170
//   ddz_sm ....................... source/RPCFKernels.cu:476-520
//   rhsNonlinear ................. source/nonlinear.cu:130-242
//   solveEq / m_multi_v .......... source/solver.cpp:107-123, matrix_op.cpp:68-78
//                                  (the time step solves the banded systems of
//                                  wallsolve.cu)
//
// The Chebyshev transforms are DCT-I of complex series: the pruned FFT of the
// even extension where the length has a plan (ydct.cuh: k_cheby_dct), else the
// block-wide FFT of the whole extension (fft.cuh: k_cheby).
#include "fftline.cuh"
#include "kernels.cuh"
#include "ydct.cuh"
#include "yline.cuh"
#include "ypass.cuh"

// ---------------------------------------------------------------------------
// Reference-layout Chebyshev transforms (drop-in cheby_s2p/p2s)
// mode 0: s2p pad (FFT length mz), 1: s2p no-pad (mz/2),
// mode 2: p2s pad (mz), 3: p2s no-pad (mz/2).
// ---------------------------------------------------------------------------
__global__ void k_cheby(PencilList in, PencilList out, long long npencils, int mode, int Ny, FftTab<double2> tab,
                        int PB, int nout) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* lines = (double2*)smem_raw;
  const int L = tab.plan.L, H = L / 2;
  const long long p0 = (long long)blockIdx.x * PB;
  for (int w = threadIdx.x; w < PB * L; w += blockDim.x) {
    const int b = w / L;
    const int n = w - b * L;
    const long long p = p0 + b;
    double2 val = make_double2(0.0, 0.0);
    if (p < npencils) {
      const double2* src = field_base<double2>(in, blockIdx.y) + p * in.ps;
      const int m = n <= H ? n : L - n;  // even extension
      if (mode == 0) {
        if (m < Ny) val = src[m] * (m ? 0.5 : 1.0);
      } else if (mode == 1) {
        val = src[m] * (m && m < H ? 0.5 : 1.0);
      } else {
        val = src[m];
      }
    }
    lines[(size_t)b * L + tab.drev[n]] = val;
  }
  fft_batch<double2, false>(lines, PB, L, tab.plan, tab.tw);
  for (int w = threadIdx.x; w < PB * nout; w += blockDim.x) {
    const int b = w / nout;
    const int k = w - b * nout;
    const long long p = p0 + b;
    if (p >= npencils) continue;
    double2 v = lines[(size_t)b * L + k];
    if (mode >= 2 && k <= H) v = v * (k && k < H ? 1.0 / H : 0.5 / H);
    (field_base<double2>(out, blockIdx.y) + p * out.ps)[k] = v;
  }
}

// Same transforms by pruned DCTs (ydct.cuh), six pencils per CTA of two
// warps; pass A reads the pencils and pass B stores them straight from and to
// global memory, with a block barrier in between (in place: every input is
// read before any output is stored).  MODE 3 = 2.  Three fields of 384 x 384 x
// 512 to points 923 -> 146 us, three of 192 x 192 x 256 to coefficients 130 ->
// 28, against one barrier and one trip through shared memory per radix 4.
template <int M, int MODE, int MB>
__global__ void __launch_bounds__(64, MB) k_cheby_dct(PencilList in, PencilList out, long long npencils, int tail,
                                                      const double2* __restrict__ dt) {
  typedef Dct<double2, M, 6> D;
  constexpr int H = M / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* X = (double2*)smem_raw;
  const long long p0 = (long long)blockIdx.x * 6;
  const int np = (int)min(6LL, npencils - p0);
  const double2* src = field_base<double2>(in, blockIdx.y) + p0 * in.ps;
  for (int i = threadIdx.x; i < D::IA; i += 64)
    D::template pass_a<MODE == 0 ? M / 4 + 1 : 0>(X, i, [&](int l, int n) {
      const double2 v = l < np ? src[l * in.ps + n] : make_double2(0.0, 0.0);
      if (MODE >= 2) return v;
      return v * (n && (MODE == 0 || n < H) ? 0.5 : 1.0);
    });
  __syncthreads();
  double2* dst = field_base<double2>(out, blockIdx.y) + p0 * out.ps;
  for (int i = threadIdx.x; i < D::IB; i += 64)
    D::pass_b(X, dt, i, [&](int l, int k, double2 v) {
      if (l >= np) return;
      double2* d = dst + l * out.ps;
      if (tail && k && k < H) d[M - k] = v;
      d[k] = MODE < 2 ? v : v * (k && k < H ? 1.0 / H : 0.5 / H);
    });
}

// ---------------------------------------------------------------------------
// getUVW on reference-layout pencils (six fields, FP64)
// ---------------------------------------------------------------------------
struct SixPtr {
  double2* f[6];  // u, v(span), w(wall), omega_x, omega_y, omega_z(wall)
  long long ps;
};

__global__ void k_get_uvw(SixPtr a, DnsGeom g, PhysParams ph) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Ny = g.Ny;
  Carve cv(smem_raw);
  double2* w = cv.take<double2>(Ny);
  double2* oz = cv.take<double2>(Ny);
  double2* Dw = cv.take<double2>(Ny);
  double2* u = cv.take<double2>(Ny);
  double2* v = cv.take<double2>(Ny);
  double2* Du = cv.take<double2>(Ny);
  double2* Dv = cv.take<double2>(Ny);
  const long long p = blockIdx.x;
  int run, kx, kz;
  pencil_modes(g, p, run, kx, kz);
  const bool zero = (kx == 0 && kz == 0);
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = kmn_of(ia, ib);
  const double kmn1 = zero ? 0.0 : 1.0 / kmn;
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    w[n] = a.f[2][p * a.ps + n];
    oz[n] = a.f[5][p * a.ps + n];
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
      // u = i(ia/k^2) Dw - i(ib/k^2) oz ; v = i(ib/k^2) Dw + i(ia/k^2) oz
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
    a.f[0][p * a.ps + n] = u[n];
    a.f[1][p * a.ps + n] = v[n];
    const double2 ox = Dv[n] - muli(wn * ib);
    const double2 oy = muli(wn * ia) - Du[n];
    a.f[3][p * a.ps + n] = ox;
    a.f[4][p * a.ps + n] = oy;
    if (zero) {
      a.f[2][p * a.ps + n] = make_double2(0.0, 0.0);
      a.f[5][p * a.ps + n] = make_double2(0.0, 0.0);
    }
  }
}

// ---------------------------------------------------------------------------
// rhsNonlinear on reference-layout pencils (FP64)
// ---------------------------------------------------------------------------
__global__ void k_rhs_nonlinear(double2* lx, double2* ly, const double2* lz, long long ps,
                                DnsGeom g, PhysParams ph) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Ny = g.Ny;
  Carve cv(smem_raw);
  double2* ax = cv.take<double2>(Ny);
  double2* ay = cv.take<double2>(Ny);
  double2* Dx = cv.take<double2>(Ny);
  double2* Dy = cv.take<double2>(Ny);
  const long long p = blockIdx.x;
  int run, kx, kz;
  pencil_modes(g, p, run, kx, kz);
  if (kx == 0 && kz == 0) return;  // source/nonlinear.cu:157
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = kmn_of(ia, ib);
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    ax[n] = lx[p * ps + n];
    ay[n] = ly[p * ps + n];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  if (warp == 0) ddz_warp(ax, Dx, Ny);
  if (warp == 1) ddz_warp(ay, Dy, Ny);
  __syncthreads();
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    const double2 hv = lz[p * ps + n] * kmn + muli(Dx[n] * ia) + muli(Dy[n] * ib);
    const double2 ho = muli(ay[n] * ia) - muli(ax[n] * ib);
    lx[p * ps + n] = hv;
    ly[p * ps + n] = ho;
  }
}

// ---------------------------------------------------------------------------
// solveEq: rhs <- inv * rhs per pencil, inverses row-major [pencil][N][N]
// (source/solver.cpp:107-123).  One warp per row, lanes over columns.
// ---------------------------------------------------------------------------
__global__ void k_solve_eq(const double2* __restrict__ inv, double2* rhs, long long ps,
                           int N, long long npencils) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* r = (double2*)smem_raw;
  double2* x = r + N;
  const long long p = blockIdx.x;
  if (p >= npencils) return;
  for (int n = threadIdx.x; n < N; n += blockDim.x) r[n] = rhs[p * ps + n];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int nw = blockDim.x >> 5;
  const double2* A = inv + p * (long long)N * N;
  for (int i = threadIdx.x >> 5; i < N; i += nw) {
    double sr = 0, si = 0;
    for (int j = lane; j < N; j += 32) {
      const double2 a = __ldg(A + (long long)i * N + j);
      const double2 b = r[j];
      sr += a.x * b.x - a.y * b.y;
      si += a.x * b.y + a.y * b.x;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      sr += __shfl_down_sync(0xffffffffu, sr, d);
      si += __shfl_down_sync(0xffffffffu, si, d);
    }
    if (lane == 0) x[i] = make_double2(sr, si);
  }
  __syncthreads();
  for (int n = threadIdx.x; n < N; n += blockDim.x) rhs[p * ps + n] = x[n];
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
cudaError_t launch_cheby(PencilList in, PencilList out, int nf, long long npencils, int mode, int Ny,
                         FftTab<double2> tab, bool tail, cudaStream_t st) {
  const int L = tab.plan.L;
  // the pruned DCT takes the zeros above Ny = L/4 + 1 as known
  if (tab.dt && (mode != 0 || Ny == L / 4 + 1)) {
    const cudaError_t e = with_len_cheby(L, [&](auto MM) -> cudaError_t {
      constexpr int M = decltype(MM)::value;
      typedef Dct<double2, M, 6> D;
      constexpr int MB = D::RA > 24 ? 4 : (D::RA > 18 ? 6 : 8);
      auto k = mode == 0 ? k_cheby_dct<M, 0, MB> : mode == 1 ? k_cheby_dct<M, 1, MB> : k_cheby_dct<M, 2, MB>;
      const size_t sm = sizeof(double2) * D::XN;
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      k<<<dim3((unsigned)((npencils + 5) / 6), nf), 64, sm, st>>>(in, out, npencils, tail, tab.dt);
      return cudaGetLastError();
    });
    if (e != cudaErrorNotSupported) return e;
  }
  int PB = (int)(32768 / ((size_t)L * 16));
  PB = PB < 1 ? 1 : (PB > 8 ? 8 : PB);
  const size_t sm = (size_t)PB * L * 16;
  cudaFuncSetAttribute(k_cheby, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_cheby<<<dim3((unsigned)((npencils + PB - 1) / PB), nf), 256, sm, st>>>(in, out, npencils, mode, Ny, tab, PB,
                                                                           tail ? L : L / 2 + 1);
  return cudaGetLastError();
}

cudaError_t launch_get_uvw(double2* const f[6], long long ps, DnsGeom g, PhysParams ph,
                           cudaStream_t st) {
  SixPtr a;
  for (int i = 0; i < 6; ++i) a.f[i] = f[i];
  a.ps = ps;
  const size_t sm = 7 * (((size_t)g.Ny * 16 + 15) & ~(size_t)15);
  cudaFuncSetAttribute(k_get_uvw, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_get_uvw<<<(unsigned)g.H, 128, sm, st>>>(a, g, ph);
  return cudaGetLastError();
}

cudaError_t launch_rhs_nonlinear(double2* lx, double2* ly, const double2* lz, long long ps,
                                 DnsGeom g, PhysParams ph, cudaStream_t st) {
  const size_t sm = 4 * (((size_t)g.Ny * 16 + 15) & ~(size_t)15);
  cudaFuncSetAttribute(k_rhs_nonlinear, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_rhs_nonlinear<<<(unsigned)g.H, 128, sm, st>>>(lx, ly, lz, ps, g, ph);
  return cudaGetLastError();
}

cudaError_t launch_solve_eq(const double2* inv, double2* rhs, long long ps, int N,
                            long long npencils, cudaStream_t st) {
  const size_t sm = (size_t)2 * N * 16;
  cudaFuncSetAttribute(k_solve_eq, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_solve_eq<<<(unsigned)npencils, 256, sm, st>>>(inv, rhs, ps, N, npencils);
  return cudaGetLastError();
}
