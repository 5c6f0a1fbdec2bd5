// Solve-only entry of the wall-normal systems: the reference's solveEq
// (source/solver.cpp:107-123) for the v and the omega_y system of every
// Fourier mode, with the banded factors of wallsolve.h in place of the
// explicit inverses (source/matrix_op.cpp:68-78).
//
// The right-hand sides arrive in the reference's collocation form
// (source/coefficient.cu:7-86): for v, rows 0..3 are the wall values v(1),
// v(-1), v'(1), v'(-1) and rows 4..N the values at the Gauss-Lobatto points
// y_2..y_{N-2}; for omega_y and for the mean modes (pencil (0,0) of both
// arrays) rows 0..1 are the wall values and rows 2..N the values at
// y_1..y_{N-1}.  Per pencil:
//   1. p = the Chebyshev polynomial of lowest degree that meets the wall rows
//      (cubic for v, linear otherwise);
//   2. f = the interior rows minus (A p) at their points, zero at the points
//      the equation leaves out, and the coefficients of its interpolant
//      (DCT-I over the Gauss-Lobatto points: the FFT of the even extension,
//      the library's no-padding p2s);
//   3. rows K .. K+n-1 of the K-fold Chebyshev integral (K = 4 for v, 2
//      otherwise), the input of the banded solve, which then runs without
//      the tilting term;
//   4. x = the banded solution + p, written over the right-hand side by the
//      solve itself.
// A p is evaluated from the operator rows of the reference's matrices:
//   v:     Re part  (1 + k^2 dt/Re) p'' - k^2 (1 + k^2 dt/(2Re)) p   (p'''' = 0)
//          Im part  a dt/2 U p'' - (k^2 a dt/2 U + a dt/2 U'') p
//   omega: (1 + k^2 dt/(2Re)) p + i a dt/2 U p                       (p'' = 0)
//   mean:  p                                                          (p'' = 0)
// with a = kx/aphi the streamwise wavenumber and k^2 = a^2 + b^2.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "wallsolve_dev.cuh"
#include "ydct.cuh"

namespace {

__device__ __forceinline__ double2 cx(double a, double b) { return make_double2(a, b); }

// 1-2. wall polynomial and the point values of the interior right-hand side
// minus A p, zero where the equation has no row; written as Gauss-Lobatto
// values (m = 0..N, pitch sp) for the DCT-I that follows
__global__ void __launch_bounds__(128) k_colloc_prep(const double2* __restrict__ bv,
                                                     const double2* __restrict__ bo, long long bp,
                                                     double2* sv, double2* so, long long sp,
                                                     double2* pbc, const double* __restrict__ cosk,
                                                     const double* __restrict__ Ut,
                                                     const double* __restrict__ ddUt, DnsGeom g,
                                                     PhysParams ph) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Ny = g.Ny, N = Ny - 1;
  const long long p = blockIdx.x;
  const int kx = (int)(p % g.Kx), kz = (int)(p / g.Kx);
  const bool zero = p == 0;
  double2* rv = (double2*)smem_raw;
  double2* ro = rv + Ny;
  __shared__ double2 pc[6];
  for (int k = threadIdx.x; k < Ny; k += blockDim.x) {
    rv[k] = bv[p * bp + k];
    ro[k] = bo[p * bp + k];
  }
  __syncthreads();
  // wall polynomial: T_j(+-1) = (+-1)^j, T_j'(1) = j^2, T_j'(-1) = (-1)^(j+1) j^2
  if (threadIdx.x == 0) {
    const double2 e = (rv[0] + rv[1]) * 0.5, o = (rv[0] - rv[1]) * 0.5;
    if (zero) {
      pc[0] = e; pc[1] = o; pc[2] = cx(0, 0); pc[3] = cx(0, 0);
    } else {
      const double2 c2 = (rv[2] - rv[3]) * 0.125;
      const double2 c3 = ((rv[2] + rv[3]) * 0.5 - o) * 0.125;
      pc[0] = e - c2; pc[1] = o - c3; pc[2] = c2; pc[3] = c3;
    }
    pc[4] = (ro[0] + ro[1]) * 0.5;
    pc[5] = (ro[0] - ro[1]) * 0.5;
    for (int j = 0; j < 6; ++j) pbc[p * 6 + j] = pc[j];
  }
  __syncthreads();
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = ia * ia + ib * ib, dt = ph.dt, Re = ph.Re;
  for (int m = threadIdx.x; m <= N; m += blockDim.x) {
    double2 fv = cx(0, 0), fo = cx(0, 0);
    const double y = __ldg(cosk + m);
    if (zero) {
      if (m >= 1 && m <= N - 1) {
        fv = rv[m + 1] - (pc[0] + pc[1] * y);
        fo = ro[m + 1] - (pc[4] + pc[5] * y);
      }
    } else {
      if (m >= 2 && m <= N - 2) {
        const double2 P0 = pc[0] + pc[1] * y + pc[2] * (2 * y * y - 1) + pc[3] * (y * (4 * y * y - 3));
        const double2 P2 = pc[2] * 4.0 + pc[3] * (24.0 * y);
        const double U = Ut[m], ddU = ddUt[m];
        const double2 re = P2 * (1 + kmn * dt / Re) - P0 * (kmn * (1 + kmn * dt * 0.5 / Re));
        const double2 im = P2 * (ia * dt * 0.5 * U) - P0 * (kmn * ia * dt * 0.5 * U + ia * dt * 0.5 * ddU);
        fv = rv[m + 2] - (re + muli(im));
      }
      if (m >= 1 && m <= N - 1) {
        const double2 P0 = pc[4] + pc[5] * y;
        fo = ro[m + 1] - (P0 * (1 + kmn * dt * 0.5 / Re) + muli(P0 * (ia * dt * 0.5 * Ut[m])));
      }
    }
    sv[p * sp + m] = fv;
    so[p * sp + m] = fo;
  }
}

// 3. rows K .. K+n-1 of the K-fold Chebyshev integral of the interpolant
// coefficients a_0..a_N (K = 4 for v, 2 for omega_y and the mean modes):
// (B x)_k = (c_{k-1} x_{k-1} - x_{k+1}) / (2k), (B x)_0 = 0
__global__ void __launch_bounds__(128) k_colloc_integrate(const double2* __restrict__ cv,
                                                          const double2* __restrict__ co, long long cp,
                                                          double2* gv, double2* go, int nv, int no,
                                                          long long gp, DnsGeom g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Ny = g.Ny, N = Ny - 1, LB = Ny + 8;
  const long long p = blockIdx.x;
  const bool zero = p == 0;
  double2* av = (double2*)smem_raw;
  double2* sv = av + LB;
  double2* ao = sv + LB;
  double2* so = ao + LB;
  for (int k = threadIdx.x; k < LB; k += blockDim.x) {
    av[k] = k <= N ? cv[p * cp + k] : cx(0, 0);
    ao[k] = k <= N ? co[p * cp + k] : cx(0, 0);
  }
  __syncthreads();
  const int Kv = zero ? 2 : 4;
  for (int it = 0; it < Kv; ++it) {
    const int nf = (it < 2) ? 2 : 1;
    for (int t = threadIdx.x; t < nf * LB; t += blockDim.x) {
      const int f = t / LB;
      const int k = t - f * LB;
      const double2* x = f ? ao : av;
      double2* y = f ? so : sv;
      double2 r = cx(0, 0);
      if (k >= 1) {
        const double2 xm = x[k - 1] * (k == 1 ? 2.0 : 1.0);
        const double2 xp = (k + 1 < LB) ? x[k + 1] : cx(0, 0);
        r = (xm - xp) * (1.0 / (2.0 * k));
      }
      y[k] = r;
    }
    __syncthreads();
    double2* tmp = av; av = sv; sv = tmp;
    if (it < 2) { tmp = ao; ao = so; so = tmp; }
  }
  for (int r = threadIdx.x; r < nv; r += blockDim.x) gv[p * gp + r] = (Kv + r < LB) ? av[Kv + r] : cx(0, 0);
  for (int r = threadIdx.x; r < no; r += blockDim.x) go[p * gp + r] = (2 + r < LB) ? ao[2 + r] : cx(0, 0);
}

// any non-finite real or imaginary part in a or b sets *flag
__global__ void __launch_bounds__(256) k_nonfinite(const double2* __restrict__ a,
                                                   const double2* __restrict__ b, long long n,
                                                   int* flag) {
  bool bad = false;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double2 x = a[i], y = b[i];
    bad |= !(isfinite(x.x) && isfinite(x.y) && isfinite(y.x) && isfinite(y.y));
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

// 1-3 fused: four lines (a system of a pencil each) per CTA of two warps.  A
// warp forms the wall polynomial and the point values of two lines of one system
// from the right-hand sides in global memory, the DCT-I over the Gauss-Lobatto points is
// a pruned one (ydct.cuh, even extension of length L = 2 N), and the K-fold
// integral its banded stencils.  A missing system has no lines.
//
// What bounds it: the whole FFT of each even extension (three passes of twice
// the points) and four integration sweeps kept a call on shared memory; now a
// value crosses it twice.  45 % of a warp's cycles then waited for L1, the tables
// among it, so two lines share each table value (23 % now, the L1 data pipe at 70 %)
// and eight CTAs an SM (six with 32-point butterflies; six, seven, eight, ten at
// 384: 451, 433, 423, 487 us before the sharing).  384 x 193 x 384: 555 -> 347 us,
// and the 140 us of a last kernel that added the wall polynomial are gone.
template <int L>
__global__ void __launch_bounds__(64, DPlan<L>::A > 24 ? 6 : 8)
                                         k_colloc_dct(const double2* __restrict__ bv, const double2* __restrict__ bo,
                                                      long long bp, double2* pbc, const double* __restrict__ Ut,
                                                      const double* __restrict__ ddUt, double2* gv, double2* go, int nv,
                                                      int no, long long gp, RhsTabs tb, DnsGeom g, PhysParams ph,
                                                      const double2* __restrict__ dt) {
  typedef Dct<double2, L, 4> D;
  constexpr int N = L / 2, Ny = N + 1, VS = Ny + 12;  // zeros above N for the stencils
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* F = (double2*)smem_raw;  // point values, then coefficients
  double2* X = F + 4 * VS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool both = bv && bo;
  const long long nlines = both ? 2 * g.H : g.H, l0 = (long long)blockIdx.x * 4;
  // a warp's lines: l0 + warp + 2 u, of one system, so that they share what is
  // read from the tables.  Both right-hand sides first, every load in flight:
  // rows m + 2 (v) or m + 1 (omega and the mean modes) at point m
  constexpr int KP = (Ny + 31) / 32;
  const bool om = both ? (warp & 1) : !bv;
  double2 row[2][KP], wall[2][4];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const long long gl = min(l0 + warp + 2 * u, nlines - (both ? 2 - warp : 1));
    const long long p = both ? gl >> 1 : gl;
    const double2* b = (om ? bo : bv) + p * bp;
    const int off = om || p == 0 ? 1 : 2;
#pragma unroll
    for (int i = 0; i < KP; ++i) row[u][i] = b[min(lane + 32 * i + off, N)];
#pragma unroll
    for (int i = 0; i < 4; ++i) wall[u][i] = b[i];
  }
  // the wavenumbers of both lines at once (lane u: line u): FP64 divisions
  double la, lb;
  {
    const long long gl = min(l0 + warp + 2 * (lane & 1), nlines - 1);
    const long long p = both ? gl >> 1 : gl;
    wavenumbers((int)(p % g.Kx), (int)(p / g.Kx), g.Nz, ph.aphi, ph.beta, la, lb);
  }
  const double h = ph.dt * 0.5 / ph.Re;
  double2 pc[2][4];
  double k2[2], ah[2];
  bool live[2], zero[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const double ia = __shfl_sync(0xffffffffu, la, u), ib = __shfl_sync(0xffffffffu, lb, u);
    const long long gl = l0 + warp + 2 * u, p = both ? gl >> 1 : gl;
    live[u] = gl < nlines;
    zero[u] = p == 0;
    k2[u] = ia * ia + ib * ib;
    ah[u] = ia * ph.dt * 0.5;
    // wall polynomial (rows 0..3 of the right-hand side)
    const double2 e = (wall[u][0] + wall[u][1]) * 0.5, o = (wall[u][0] - wall[u][1]) * 0.5;
    pc[u][0] = e;
    pc[u][1] = o;
    pc[u][2] = pc[u][3] = cx(0, 0);
    if (!om && !zero[u]) {
      pc[u][2] = (wall[u][2] - wall[u][3]) * 0.125;
      pc[u][3] = ((wall[u][2] + wall[u][3]) * 0.5 - o) * 0.125;
      pc[u][0] = e - pc[u][2];
      pc[u][1] = o - pc[u][3];
    }
    if (lane == 0 && live[u]) {
      double2* q = pbc + p * 6 + (om ? 4 : 0);
      q[0] = pc[u][0];
      q[1] = pc[u][1];
      if (!om) { q[2] = pc[u][2]; q[3] = pc[u][3]; }
    }
  }
  // point value m of the interior right-hand side minus A p, zero where the
  // equation has no row
#pragma unroll
  for (int i = 0; i < KP; ++i) {
    const int m = lane + 32 * i;
    if (m > N) break;
    const double y = __ldg(tb.cosk + m), U = __ldg(Ut + m), ddU = om ? 0.0 : __ldg(ddUt + m);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      double2 v = cx(0, 0);
      if (om || zero[u]) {
        if (m >= 1 && m <= N - 1) {
          const double2 P0 = pc[u][0] + pc[u][1] * y;
          v = zero[u] ? row[u][i] - P0 : row[u][i] - (P0 * (1 + k2[u] * h) + muli(P0 * (ah[u] * U)));
        }
      } else if (m >= 2 && m <= N - 2) {
        const double2 P0 = pc[u][0] + pc[u][1] * y + pc[u][2] * (2 * y * y - 1) + pc[u][3] * (y * (4 * y * y - 3));
        const double2 P2 = pc[u][2] * 4.0 + pc[u][3] * (24.0 * y);
        const double cv2 = 1 + 2.0 * k2[u] * h, cv0 = k2[u] * (1 + k2[u] * h);
        const double2 re = P2 * cv2 - P0 * cv0;
        const double2 im = P2 * (ah[u] * U) - P0 * (k2[u] * ah[u] * U + ah[u] * ddU);
        v = row[u][i] - (re + muli(im));
      }
      F[(warp + 2 * u) * VS + m] = live[u] ? v : cx(0, 0);
    }
  }
  for (int i = threadIdx.x; i < 4 * 12; i += 64) F[i / 12 * VS + Ny + i % 12] = cx(0, 0);
  __syncthreads();
  for (int i = threadIdx.x; i < D::IA; i += 64)
    D::template pass_a<0>(X, i, [&](int l, int n) { return F[l * VS + n]; });
  __syncthreads();
  for (int i = threadIdx.x; i < D::IB; i += 64)
    D::pass_b(X, dt, i, [&](int l, int k, double2 v) { F[l * VS + k] = v * (k && k < N ? 1.0 / N : 0.5 / N); });
  __syncthreads();
  // rows K .. K+n-1 of the K-fold integral (K = 4 for v, 2 otherwise)
  const double2 *f0 = F + warp * VS, *f1 = f0 + 2 * VS;
  double2* out = (om ? go : gv) + (both ? l0 >> 1 : l0 + warp) * gp;
  const long long step = (both ? 1 : 2) * gp;  // to the warp's second line
  if (om) {
#pragma unroll 2
    for (int r = lane; r < nv; r += 32) {  // (as many rows of omega)
      double2 v0 = cx(0, 0), v1 = cx(0, 0);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double w = __ldg(tb.b2 + d * (nv + 2) + r);
        v0 = v0 + f0[r + 2 * d] * w;
        v1 = v1 + f1[r + 2 * d] * w;
      }
      if (live[0]) out[r] = v0;
      if (live[1]) out[step + r] = v1;
    }
  } else {
#pragma unroll 2
    for (int r = lane; r < nv; r += 32) {
      double2 v0 = cx(0, 0), v1 = cx(0, 0);
#pragma unroll
      for (int d = 0; d < 5; ++d) {
        const double w = __ldg(tb.b4 + d * nv + r);
        v0 = v0 + f0[r + 2 * d] * w;
        v1 = v1 + f1[r + 2 * d] * w;
      }
      if (zero[0]) {  // the mean modes: two-fold
        v0 = cx(0, 0);
#pragma unroll
        for (int d = 0; d < 3; ++d) v0 = v0 + f0[r + 2 * d] * __ldg(tb.b2 + d * (nv + 2) + r);
      }
      if (live[0]) out[r] = v0;
      if (live[1]) out[step + r] = v1;
    }
  }
}

}  // namespace

cudaError_t launch_nonfinite(const double2* a, const double2* b, long long n, int* flag,
                             cudaStream_t st) {
  const long long blocks = std::min<long long>((n + 255) / 256, 148LL * 8);
  k_nonfinite<<<(unsigned)std::max<long long>(blocks, 1), 256, 0, st>>>(a, b, n, flag);
  return cudaGetLastError();
}

cudaError_t launch_colloc_prep(const double2* bv, const double2* bo, long long bp, double2* sv,
                               double2* so, long long sp, double2* pbc, const double* cosk,
                               const double* Ut, const double* ddUt, const DnsGeom& g,
                               const PhysParams& ph, cudaStream_t st) {
  const size_t sm = (size_t)32 * g.Ny;
  if (sm > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_colloc_prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e) return e;
  }
  k_colloc_prep<<<(unsigned)g.H, 128, sm, st>>>(bv, bo, bp, sv, so, sp, pbc, cosk, Ut, ddUt, g, ph);
  return cudaGetLastError();
}

cudaError_t launch_colloc_integrate(const double2* cv, const double2* co, long long cp, double2* gv,
                                    double2* go, const WallDims& wd, const DnsGeom& g, cudaStream_t st) {
  const size_t sm = (size_t)64 * (g.Ny + 8);
  if (sm > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_colloc_integrate, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e) return e;
  }
  k_colloc_integrate<<<(unsigned)g.H, 128, sm, st>>>(cv, co, cp, gv, go, wd.nv, wd.no, wd.gp, g);
  return cudaGetLastError();
}

cudaError_t launch_colloc_fused(const double2* bv, const double2* bo, long long bp, double2* pbc,
                                const double* Ut, const double* ddUt, double2* gv, double2* go, const WallDims& wd,
                                const RhsTabs& tb, const DnsGeom& g, const PhysParams& ph, FftTab<double2> tab,
                                cudaStream_t st) {
  if (!tab.dt || g.Ny != tab.plan.L / 2 + 1 || wd.nv != wd.no) return cudaErrorNotSupported;
  return with_len_cheby(tab.plan.L, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    const size_t sm = (size_t)(4 * (L / 2 + 13) + Dct<double2, L, 4>::XN) * 16;
    const long long nlines = bv && bo ? 2 * g.H : g.H;
    auto k = k_colloc_dct<L>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<(unsigned)((nlines + 3) / 4), 64, sm, st>>>(bv, bo, bp, pbc, Ut, ddUt, gv, go, wd.nv, wd.no, wd.gp, tb, g, ph,
                                                    tab.dt);
    return cudaGetLastError();
  });
}
