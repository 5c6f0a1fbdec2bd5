// Reference-layout right-hand sides of the Crank-Nicolson / AB2 step, for
// callers that run the reference's step sequence function by function
// (get_rhs_v -> solveEq -> get_rhs_omega -> solveEq):
//
//   dns_rhs_v ......... get_linear_v + the AB2 loop of get_rhs_v
//                       (source/linear.cpp:7-41,86-125, source/rhs.cpp:185-219)
//   dns_rhs_omega ..... get_linear_omega_y (source/linear.cpp:52-84,127-171)
//   dns_rhs_mean ...... get_linear_zero_wave_u_w (source/linear.cpp:43-50,173-205)
//   dns_operator_tables / dns_operator_matrices ... the T matrices, U profile
//                       and collocation operators initAuxMatrix stores
//                       (source/solver.cpp:260-320, source/coefficient.cu)
//
// The fused time step does not use these kernels: it forms the same right-
// hand sides in Chebyshev coefficient space inside its y1 pass.  Here each
// pencil's right-hand side is the reference's collocation form, evaluated on
// the GPU, FP64 throughout: in coefficient space (derivatives by sweeps,
// products with U and U' as interpolants) and one DCT-I to the points
// (k_rhs_dct), or, for lengths without a DCT plan, as products with the T
// tables, one warp per collocation row.
#include <algorithm>
#include <string>

#include "../../include/dns_b200.h"
#include "context_impl.cuh"
#include "ycoef.cuh"
#include "ydct.cuh"

namespace {

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double2 warp_sum(double2 v) {
  return make_double2(warp_sum(v.x), warp_sum(v.y));
}

// rows 4..N: the explicit half of the CN v operator applied to v^n at the
// collocation point r = i - 2, plus AB2; rows 0..3 (wall rows) zero; v^n is
// saved to rvp (the reference's rhs_v_p).  Pencil (0,0) is left alone.
__global__ void k_rhs_v(double2* rv, double2* rvp, const double2* nv, const double2* nvp,
                        long long ps, const double* T0, const double* T2, const double* T4,
                        const double* U, const double* ddU, DnsGeom g, PhysParams ph) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* v = (double2*)smem_raw;
  const int Ny = g.Ny;
  const long long p = blockIdx.x;
  const int kx = (int)(p % g.Kx), kz = (int)(p / g.Kx);
  if (kx == 0 && kz == 0) return;
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = kmn_of(ia, ib);
  const double dt = ph.dt, Re = ph.Re;
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    v[n] = rv[p * ps + n];
    rvp[p * ps + n] = v[n];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double a4 = dt * 0.5 / Re, a2 = 1 - kmn * dt / Re, a0 = -kmn * (1 - kmn * dt * 0.5 / Re);
  for (int i = warp; i < Ny; i += nw) {
    double2 out = make_double2(0.0, 0.0);
    if (i >= 4) {
      const int r = i - 2;
      double2 P0 = make_double2(0, 0), P2 = P0, P4 = P0;
      for (int j = lane; j < Ny; j += 32) {
        const size_t c = (size_t)r * Ny + j;
        P0 = P0 + v[j] * T0[c];
        P2 = P2 + v[j] * T2[c];
        P4 = P4 + v[j] * T4[c];
      }
      P0 = warp_sum(P0);
      P2 = warp_sum(P2);
      P4 = warp_sum(P4);
      const double b2 = -ia * dt * 0.5 * U[r];
      const double b0 = kmn * ia * dt * 0.5 * U[r] + ia * dt * 0.5 * ddU[r];
      out = P4 * a4 + P2 * a2 + P0 * a0 + muli(P2 * b2 + P0 * b0);
      out = out + (nv[p * ps + r] * 1.5 - nvp[p * ps + r] * 0.5) * dt;
    }
    if (lane == 0) rv[p * ps + i] = out;
  }
}

// rows 2..N: the explicit half of the CN omega operator at r = i - 1, the
// tilting term -i beta U' dt/2 (v^{n+1} + v^n) and AB2; rows 0, 1 zero.
__global__ void k_rhs_omega(double2* ro, const double2* no, const double2* nop, const double2* vn1,
                            const double2* vn, long long ps, const double* T0, const double* T2,
                            const double* U, const double* dU, DnsGeom g, PhysParams ph) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* o = (double2*)smem_raw;
  double2* s = o + g.Ny;
  const int Ny = g.Ny;
  const long long p = blockIdx.x;
  const int kx = (int)(p % g.Kx), kz = (int)(p / g.Kx);
  if (kx == 0 && kz == 0) return;
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kmn = kmn_of(ia, ib);
  const double dt = ph.dt, Re = ph.Re;
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) {
    o[n] = ro[p * ps + n];
    s[n] = vn[p * ps + n] + vn1[p * ps + n];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double a2 = 0.5 / Re * dt, a0 = 1 - kmn * dt * 0.5 / Re;
  for (int i = warp; i < Ny; i += nw) {
    double2 out = make_double2(0.0, 0.0);
    if (i >= 2) {
      const int r = i - 1;
      double2 Q0 = make_double2(0, 0), Q2 = Q0, S0 = Q0;
      for (int j = lane; j < Ny; j += 32) {
        const size_t c = (size_t)r * Ny + j;
        Q0 = Q0 + o[j] * T0[c];
        Q2 = Q2 + o[j] * T2[c];
        S0 = S0 + s[j] * T0[c];
      }
      Q0 = warp_sum(Q0);
      Q2 = warp_sum(Q2);
      S0 = warp_sum(S0);
      out = Q2 * a2 + Q0 * a0 + muli(Q0 * (-ia * dt * 0.5 * U[r]) + S0 * (-0.5 * ib * dU[r] * dt));
      out = out + (no[p * ps + r] * 1.5 - nop[p * ps + r] * 0.5) * dt;
    }
    if (lane == 0) ro[p * ps + i] = out;
  }
}

// Both right-hand sides of a pencil through one DCT-I over the Gauss-Lobatto
// points (even extension of length L = 2 N): four pencils per CTA, a warp
// each for the coefficients.  OMEGA = false: k_rhs_v, true: k_rhs_omega.
//
// What bounds it: the T-table form reads three Ny x Ny tables through L1 for
// every pencil, 2 Ny^2 products each; here a pencil's vectors are read and
// written once.  128 x 65 x 128, v / omega_y: 202 / 221 -> 36 / 30 us.
template <int L, bool OMEGA>
__global__ void __launch_bounds__(128) k_rhs_dct(double2* x, double2* xp, const double2* nl, const double2* nlp,
                                                 const double2* vn1, const double2* vn, long long ps, DnsGeom g,
                                                 PhysParams ph, const double2* __restrict__ dt) {
  typedef Dct<double2, L, 4> D;
  constexpr int N = L / 2, Ny = N + 1, VS = Ny + 4;  // two zeros on either side
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2* A = (double2*)smem_raw + (size_t)warp * 3 * VS + 2;  // v or omega
  double2* B = A + VS;                                          // D^2 v, or the sum of the two v
  double2* F = B + VS;                                          // D^4 v or D^2 omega, then the right-hand side
  double2* X = (double2*)smem_raw + (size_t)4 * 3 * VS;
  const long long p0 = (long long)blockIdx.x * 4, p = p0 + warp;
  const double2 z2 = make_double2(0.0, 0.0);
  if (lane < 2) A[lane - 2] = A[Ny + lane] = B[lane - 2] = B[Ny + lane] = z2;
  if (p < g.H) {
    const int kx = (int)(p % g.Kx), kz = (int)(p / g.Kx);
    for (int n = lane; n < Ny; n += 32) {
      const double2 v = x[p * ps + n];
      A[n] = v;
      if (OMEGA) B[n] = vn[p * ps + n] + vn1[p * ps + n];
      else if (p) xp[p * ps + n] = v;
    }
    __syncwarp();
    double ia, ib;
    wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
    const double kmn = kmn_of(ia, ib), h = ph.dt * 0.5 / ph.Re, gam = ia * ph.dt * 0.5;
    constexpr int CH = ddz_run(Ny);
    if (OMEGA) {
      d2z_fast<CH>(A, F, Ny);
      __syncwarp();
      const double a0 = 1 - kmn * h, kap = -0.5 * ib * ph.dt;
      for (int k = lane; k < Ny; k += 32) {
        double2 P, Pf;
        u_times(A, k, N, ph, P, Pf);
        F[k] = F[k] * h + A[k] * a0 + muli(up_times(B, k, N, ph) * kap - Pf * gam);
      }
    } else {
      d2z_fast<CH>(A, B, Ny);
      __syncwarp();
      d2z_fast<CH>(B, F, Ny);
      __syncwarp();
      const double a2 = 1 - 2.0 * kmn * h, a0 = kmn * (1 - kmn * h);
      for (int k = lane; k < Ny; k += 32) {
        const double2 v = A[k], d2 = B[k];
        F[k] = F[k] * h + d2 * a2 - v * a0 + muli(v) * (2.0 * gam * ph.U2);
        B[k] = v * kmn - d2;  // under i gam U
      }
      __syncwarp();
      for (int k = lane; k < Ny; k += 32) {
        double2 P, Pf;
        u_times(B, k, N, ph, P, Pf);
        F[k] = F[k] + muli(Pf) * gam;
      }
    }
  } else {
    for (int n = lane; n < Ny; n += 32) F[n] = z2;
  }
  __syncthreads();
  const double2* F0 = (const double2*)smem_raw + 2 + 2 * VS;
  for (int i = threadIdx.x; i < D::IA; i += 128)
    D::template pass_a<0>(X, i, [&](int l, int n) { return F0[l * 3 * VS + n] * (n && n < N ? 0.5 : 1.0); });
  __syncthreads();
  // point r goes to row r + 2 (v, r = 2..N-2) or r + 1 (omega, r = 1..N-1);
  // the wall rows are zero
  constexpr int OFF = OMEGA ? 1 : 2;
  for (int i = threadIdx.x; i < D::IB; i += 128)
    D::pass_b(X, dt, i, [&](int l, int r, double2 f) {
      const long long q = p0 + l;
      if (q >= g.H || q == 0) return;
      double2* row = x + q * ps;
      if (r >= OFF && r <= N - OFF)
        row[r + OFF] = f + (nl[q * ps + r] * 1.5 - nlp[q * ps + r] * 0.5) * ph.dt;
      if (r < 2 * OFF) row[r] = z2;
    });
}

// the mean modes u0 (block 0) and w0 (block 1): rows 2..N of
// (T0 + dt/(2 Re) T2) x - dt (1.5 lambda - 0.5 lambda_p) at r = i - 1;
// rows 0, 1 (Dirichlet) zero.  Two pencils, each in place, so two blocks: a warp
// a row at a time, as many warps as there are rows or fit (a row is one latency).
__global__ void __launch_bounds__(1024) k_rhs_mean(double2* u0, const double2* lx, const double2* lxp, double2* w0,
                           const double2* lz, const double2* lzp, int Ny, const double* T0,
                           const double* T2, double Re, double dt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* x = (double2*)smem_raw;
  double2* vec = blockIdx.x == 0 ? u0 : w0;
  const double2* l = blockIdx.x == 0 ? lx : lz;
  const double2* lp = blockIdx.x == 0 ? lxp : lzp;
  for (int n = threadIdx.x; n < Ny; n += blockDim.x) x[n] = vec[n];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = warp; i < Ny; i += nw) {
    double2 out = make_double2(0.0, 0.0);
    if (i >= 2) {
      const int r = i - 1;
      double2 a = make_double2(0, 0);
      for (int j = lane; j < Ny; j += 32) {
        const size_t c = (size_t)r * Ny + j;
        a = a + x[j] * (T0[c] + dt * 0.5 / Re * T2[c]);
      }
      a = warp_sum(a);
      out = a - (l[r] * 1.5 - lp[r] * 0.5) * dt;
    }
    if (lane == 0) vec[i] = out;
  }
}

struct Stage {
  // a pencil field of the caller: pointer, read by the kernel, written by it
  const void* src;
  bool in, out;
};

// Run `launch(ptrs, ps)` on the caller's pencils: in place for device
// buffers, through the context's staging vectors (pitch Ny) for host ones.
template <typename F>
dns_status staged(dns_ctx* c, Stage* f, int n, size_t tpitch, int where, F launch) {
  const DnsGeom& g = c->g;
  const size_t row = (size_t)g.Ny * 16;
  if (where != DNS_HOST && where != DNS_DEVICE)
    return dns_internal_fail(DNS_ERR_ARG, "where must be DNS_HOST or DNS_DEVICE");
  if (tpitch % 16 || tpitch < row)
    return dns_internal_fail(DNS_ERR_ARG, "tpitch must be a multiple of 16 and hold Ny complex values");
  if (cudaSetDevice(c->P.device)) return dns_internal_fail(DNS_ERR_CUDA, "cudaSetDevice");
  double2* ptr[6];
  if (where == DNS_DEVICE) {
    for (int i = 0; i < n; ++i) ptr[i] = (double2*)f[i].src;
    cudaError_t e = launch(ptr, (long long)(tpitch / 16));
    if (e) return dns_internal_fail(DNS_ERR_CUDA, cudaGetErrorString(e));
    return DNS_OK;
  }
  const size_t hn = (size_t)g.H * g.Ny;
  if (!c->rhs_io && c->alloc(&c->rhs_io, 6 * hn))
    return dns_internal_fail(DNS_ERR_CUDA, "staging allocation");
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < n && !e; ++i) {
    ptr[i] = c->rhs_io + i * hn;
    if (f[i].in)
      e = cudaMemcpy2DAsync(ptr[i], row, f[i].src, tpitch, row, g.H, cudaMemcpyHostToDevice, c->st);
  }
  if (!e) e = launch(ptr, (long long)g.Ny);
  for (int i = 0; i < n && !e; ++i)
    if (f[i].out)
      e = cudaMemcpy2DAsync((void*)f[i].src, tpitch, ptr[i], row, row, g.H, cudaMemcpyDeviceToHost, c->st);
  if (!e) e = cudaStreamSynchronize(c->st);
  if (e) return dns_internal_fail(DNS_ERR_CUDA, cudaGetErrorString(e));
  return DNS_OK;
}

template <bool OMEGA>
cudaError_t launch_rhs_dct(dns_ctx* c, double2* x, double2* xp, const double2* nl, const double2* nlp,
                           const double2* vn1, const double2* vn, long long ps) {
  const FftTab<double2> tab = c->fy0_d.tab();
  if (!tab.dt || c->g.Ny != tab.plan.L / 2 + 1) return cudaErrorNotSupported;
  return with_len_cheby(tab.plan.L, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    auto k = k_rhs_dct<L, OMEGA>;
    const size_t sm = (size_t)(4 * 3 * (L / 2 + 5) + Dct<double2, L, 4>::XN) * 16;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<(unsigned)((c->g.H + 3) / 4), 128, sm, c->st>>>(x, xp, nl, nlp, vn1, vn, ps, c->g, c->ph, tab.dt);
    return cudaGetLastError();
  });
}

unsigned threads_for(int Ny) { return (unsigned)std::min(256, std::max(64, (Ny + 31) / 32 * 32)); }

}  // namespace

extern "C" {

dns_status dns_rhs_v(dns_ctx* c, void* rhs_v, void* rhs_v_p, const void* nv, const void* nv_p,
                     size_t tpitch, int where) {
  if (!c || !rhs_v || !rhs_v_p || !nv || !nv_p) return dns_internal_fail(DNS_ERR_ARG, "null argument");
  // rhs_v_p is copied in too: pencil (0,0) keeps its value
  Stage f[4] = {{rhs_v, true, true}, {rhs_v_p, true, true}, {nv, true, false}, {nv_p, true, false}};
  const DnsGeom g = c->g;
  const PhysParams ph = c->ph;
  const size_t sm = (size_t)g.Ny * 16;
  return staged(c, f, 4, tpitch, where, [&](double2** q, long long ps) {
    const cudaError_t e = launch_rhs_dct<false>(c, q[0], q[1], q[2], q[3], nullptr, nullptr, ps);
    if (e != cudaErrorNotSupported) return e;
    k_rhs_v<<<(unsigned)g.H, threads_for(g.Ny), sm, c->st>>>(q[0], q[1], q[2], q[3], ps, c->T0, c->T2,
                                                            c->T4, c->Ut, c->ddUt, g, ph);
    return cudaGetLastError();
  });
}

dns_status dns_rhs_omega(dns_ctx* c, void* rhs_omega, const void* nomega, const void* nomega_p,
                         const void* rhs_v, const void* rhs_v_p, size_t tpitch, int where) {
  if (!c || !rhs_omega || !nomega || !nomega_p || !rhs_v || !rhs_v_p)
    return dns_internal_fail(DNS_ERR_ARG, "null argument");
  Stage f[5] = {{rhs_omega, true, true}, {nomega, true, false}, {nomega_p, true, false},
                {rhs_v, true, false}, {rhs_v_p, true, false}};
  const DnsGeom g = c->g;
  const PhysParams ph = c->ph;
  const size_t sm = (size_t)2 * g.Ny * 16;
  return staged(c, f, 5, tpitch, where, [&](double2** q, long long ps) {
    const cudaError_t e = launch_rhs_dct<true>(c, q[0], nullptr, q[1], q[2], q[3], q[4], ps);
    if (e != cudaErrorNotSupported) return e;
    k_rhs_omega<<<(unsigned)g.H, threads_for(g.Ny), sm, c->st>>>(q[0], q[1], q[2], q[3], q[4], ps,
                                                                c->T0, c->T2, c->Ut, c->dUt, g, ph);
    return cudaGetLastError();
  });
}

dns_status dns_rhs_mean(dns_ctx* c, void* u0, const void* lambx0, const void* lambx0_p, void* w0,
                        const void* lambz0, const void* lambz0_p, int where) {
  if (!c || !u0 || !lambx0 || !lambx0_p || !w0 || !lambz0 || !lambz0_p)
    return dns_internal_fail(DNS_ERR_ARG, "null argument");
  if (where != DNS_HOST && where != DNS_DEVICE)
    return dns_internal_fail(DNS_ERR_ARG, "where must be DNS_HOST or DNS_DEVICE");
  if (cudaSetDevice(c->P.device)) return dns_internal_fail(DNS_ERR_CUDA, "cudaSetDevice");
  const int Ny = c->g.Ny;
  const size_t vb = (size_t)Ny * 16;
  const void* src[6] = {u0, lambx0, lambx0_p, w0, lambz0, lambz0_p};
  double2* q[6];
  cudaError_t e = cudaSuccess;
  if (where == DNS_HOST) {
    const size_t hn = (size_t)c->g.H * Ny;
    if (!c->rhs_io && c->alloc(&c->rhs_io, 6 * hn))
      return dns_internal_fail(DNS_ERR_CUDA, "staging allocation");
    for (int i = 0; i < 6 && !e; ++i) {
      q[i] = c->rhs_io + (size_t)i * Ny;
      e = cudaMemcpyAsync(q[i], src[i], vb, cudaMemcpyHostToDevice, c->st);
    }
  } else {
    for (int i = 0; i < 6; ++i) q[i] = (double2*)src[i];
  }
  if (!e) {
    k_rhs_mean<<<2, std::min(1024, 32 * Ny), vb, c->st>>>(q[0], q[1], q[2], q[3], q[4], q[5], Ny, c->T0, c->T2,
                                                c->ph.Re, c->ph.dt);
    e = cudaGetLastError();
  }
  if (!e && where == DNS_HOST) {
    e = cudaMemcpyAsync(u0, q[0], vb, cudaMemcpyDeviceToHost, c->st);
    if (!e) e = cudaMemcpyAsync(w0, q[3], vb, cudaMemcpyDeviceToHost, c->st);
    if (!e) e = cudaStreamSynchronize(c->st);
  }
  if (e) return dns_internal_fail(DNS_ERR_CUDA, cudaGetErrorString(e));
  return DNS_OK;
}

dns_status dns_operator_tables(dns_ctx* c, double* T0, double* T2, double* T4, double* U, double* dU,
                               double* ddU) {
  if (!c) return dns_internal_fail(DNS_ERR_ARG, "null context");
  if (cudaSetDevice(c->P.device)) return dns_internal_fail(DNS_ERR_CUDA, "cudaSetDevice");
  const size_t Ny = (size_t)c->g.Ny;
  struct { void* dst; const double* src; size_t n; } cp[6] = {
      {T0, c->T0, Ny * Ny}, {T2, c->T2, Ny * Ny}, {T4, c->T4, Ny * Ny},
      {U, c->Ut, Ny}, {dU, c->dUt, Ny}, {ddU, c->ddUt, Ny}};
  for (auto& x : cp)
    if (x.dst && cudaMemcpy(x.dst, x.src, x.n * 8, cudaMemcpyDeviceToHost))
      return dns_internal_fail(DNS_ERR_CUDA, "table copy");
  return DNS_OK;
}

}  // extern "C"
