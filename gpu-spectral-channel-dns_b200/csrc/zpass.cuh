// Spanwise (z) passes as two register butterflies around one exchange.
//
// A CTA owns TX streamwise modes x TY wall-normal points, NL = TX TY lines of
// length L = RA RB.  Pass A reads its RA inputs of a line straight from
// global memory (zero padding and the zeroed Nyquist modes are skipped
// there), pass B stores its RB outputs straight to global memory, and the
// lines cross shared memory once in between, [position][line]: the lanes of
// a warp cover whole positions, so every shared access is a run of
// consecutive addresses without padding.  Neither pass works in place, so a
// thread may take any number of butterflies of a pass, with one block barrier
// in all.
//
// What bounds it: the pass is a transpose with a transform on the way, so HBM
// should; warp-synchronous in-place lines moved each value through shared
// memory eight times (FP64, three passes and the staging), which at 128 bytes
// a clock and SM was the bound.  TY elements of a pencil and TX of a row are
// the contiguous runs, whole 32-byte sectors on both sides.
#pragma once
#include <type_traits>
#include <vector>

#include "fft2.cuh"
#include "kernels.cuh"

// radices of a length: two factors, both small enough for registers (FP64: a
// butterfly of radix R holds 4 R of them), the larger first
template <int L> struct ZPlan { enum { ok = 0, A = 1, B = 1 }; };
#define ZPLAN(L, RA, RB) \
  template <> struct ZPlan<L> { enum { ok = 1, A = RA, B = RB }; static_assert(RA * RB == L, "plan"); };
ZPLAN(24, 6, 4)
ZPLAN(32, 8, 4)
ZPLAN(36, 6, 6)
ZPLAN(48, 8, 6)
ZPLAN(54, 9, 6)
ZPLAN(64, 8, 8)
ZPLAN(72, 9, 8)
ZPLAN(96, 12, 8)
ZPLAN(108, 12, 9)
ZPLAN(128, 16, 8)
ZPLAN(144, 12, 12)
ZPLAN(162, 18, 9)
ZPLAN(192, 16, 12)
ZPLAN(216, 18, 12)
ZPLAN(256, 16, 16)
ZPLAN(288, 18, 16)
ZPLAN(324, 18, 18)
ZPLAN(384, 24, 16)
ZPLAN(432, 24, 18)
ZPLAN(512, 32, 16)
ZPLAN(576, 24, 24)
ZPLAN(768, 32, 24)
#undef ZPLAN
#define ZPLAN_LENGTHS(X) \
  X(24) X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) X(216) X(256) X(288) \
  X(324) X(384) X(432) X(512) X(576) X(768)

// Pass-B twiddles W_L^{r k}, r = 1..RB-1, k < RA, stored [r - 1][k]; W: the
// table W_L^j, j < L
template <typename C> int ztw_table(int L, const double2* W, std::vector<C>& out) {
  int ra = 0, rb = 0;
#define ZCASE(n) \
  case n: ra = ZPlan<n>::A; rb = ZPlan<n>::B; break;
  switch (L) { ZPLAN_LENGTHS(ZCASE) default: return -1; }
#undef ZCASE
  out.resize((size_t)(rb - 1) * ra);
  for (int r = 1; r < rb; ++r)
    for (int k = 0; k < ra; ++k) out[(size_t)(r - 1) * ra + k] = from_d2<C>(W[r * k]);
  return (int)out.size();
}

// The tensor-staged FP32 form (k_zbt, k_zft): a warp's pair of lines.  Element
// pos of line l sits at 2 (pos + pos / RA) + l, a pair is WS elements; before
// that the values, [n][line], lie from the pair's first 128-byte boundary on.
// Tiled copies need destinations on 128-byte boundaries and boxes of at most 256
// rows: a line up to 256 points comes in one copy, a longer one in two halves
// where the second starts on such a boundary (L a multiple of 16).
template <typename C, int L> struct ZStage {
  static constexpr int RA = ZPlan<L>::A, RB = ZPlan<L>::B;
  static constexpr int raw = 2 * RB * (RA + 1);
  static constexpr int WS = raw + (18 - raw % 16) % 16;  // 2 mod 16
  static constexpr bool ok = ZPlan<L>::ok && RB <= 16 && sizeof(C) == 8;
  static constexpr bool fits(int n) { return n * 16 + 128 <= WS * 8; }
  static constexpr int ROWS = L <= 256 ? L : L / 2;  // of a forward copy
  static constexpr bool copies_ok = ROWS <= 256 && L % ROWS == 0 && (ROWS == L || ROWS * 2 * sizeof(C) % 128 == 0);
};

#ifdef __CUDACC__
// butterfly (line li, j) of pass A after its inputs: the RA-point transform,
// outputs to positions j RA + r
template <typename C, int RA, int NL, bool INV>
__device__ __forceinline__ void zpass_a(C* v, C* buf, int li, int j) {
  Codelet<RA, INV, C>::run(v);
  C* o = buf + j * (RA * NL) + li;
#pragma unroll
  for (int r = 0; r < RA; ++r) o[r * NL] = v[r];
}
// butterfly (li, k) of pass B: positions k + r RA in and out, v on return
template <typename C, int RA, int RB, int NL, bool INV>
__device__ __forceinline__ void zpass_b(C* v, const C* buf, const C* __restrict__ tw, int li, int k) {
  const C* x = buf + k * NL + li;
#pragma unroll
  for (int r = 0; r < RB; ++r) v[r] = x[r * (RA * NL)];
#pragma unroll
  for (int r = 1; r < RB; ++r) {
    const C w = tw[(r - 1) * RA + k];
    v[r] = INV ? cmulc(v[r], w) : cmul(v[r], w);
  }
  Codelet<RB, INV, C>::run(v);
}

// spanwise inverse: pencils [f][kz Kx + kx][y] -> rows [f][y][zp][kx].  The
// streamwise Nyquist column (kx = Kx - 1) is zero and no streamwise pass reads
// it: it is left out.
template <typename C, int L, int TX, int TY, int NT, int MB, class PA>
__global__ void __launch_bounds__(NT, MB) k_zb2(PA in, RowArr out, DnsGeom g, const C* __restrict__ tw) {
  constexpr int RA = ZPlan<L>::A, RB = ZPlan<L>::B, NL = TX * TY;
  constexpr int Nz = L / 3 * 2, hz = Nz / 2;  // the launcher checks g.Nz
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = (C*)smem_raw;
  const int Kx = g.Kx, Py = g.Py;
  const int kx0 = blockIdx.x * TX, y0 = blockIdx.y * TY, f = blockIdx.z;
  const long long kzs = (long long)Kx * in.ps;
  for (int t = threadIdx.x; t < NL * RB; t += NT) {
    const int li = t % NL, j = t / NL;  // li = kxl TY + yl: TY neighbours of a pencil
    const int kx = kx0 + li / TY, y = y0 + li % TY;
    const bool ok = kx < Kx - 1 && y < Py;
    const C* src = field_base<C>(in, f) + (long long)kx * in.ps + y + (long long)j * kzs;
    C v[RA];
#pragma unroll
    for (int r = 0; r < RA; ++r) {
      // element n = j + r RB: modes kz < Nz/2, zeros, modes kz - Nz > -Nz/2
      const int n = j + r * RB;
      v[r] = cmk<C>(0.0, 0.0);
      if (r * RB < hz) {
        if (ok && n < hz) v[r] = src[(long long)(r * RB) * kzs];
      }
      if (r * RB + RB - 1 > L - hz) {
        if (ok && n > L - hz) v[r] = src[(long long)(r * RB - (L - Nz)) * kzs];
      }
    }
    zpass_a<C, RA, NL, true>(v, buf, li, j);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < NL * RA; t += NT) {
    const int li = t % NL, k = t / NL;
    C v[RB];
    zpass_b<C, RA, RB, NL, true>(v, buf, tw, li, k);
    const int kx = kx0 + li / TY, y = y0 + li % TY;
    if (kx < Kx - 1 && y < Py) {
      C* dst = (C*)out.base + (long long)f * out.fs + ((long long)y * L + k) * out.rs + kx;
#pragma unroll
      for (int r = 0; r < RB; ++r) dst[(long long)(r * RA) * out.rs] = v[r];
    }
  }
}

// spanwise forward: rows [f][y][zp][kx] -> pencils [f][kz Kx + kx][y], the
// Nz kept wavenumbers
template <typename C, int L, int TX, int TY, int NT, int MB, class PA>
__global__ void __launch_bounds__(NT, MB) k_zf2(RowArr in, PA out, DnsGeom g, const C* __restrict__ tw) {
  constexpr int RA = ZPlan<L>::A, RB = ZPlan<L>::B, NL = TX * TY;
  constexpr int Nz = L / 3 * 2, hz = Nz / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = (C*)smem_raw;
  const int Kx = g.Kx, Py = g.Py;
  const int kx0 = blockIdx.x * TX, y0 = blockIdx.y * TY, f = blockIdx.z;
  for (int t = threadIdx.x; t < NL * RB; t += NT) {
    const int li = t % NL, j = t / NL;
    const int kx = kx0 + li / TY, y = y0 + li % TY;
    const bool ok = kx < Kx && y < Py;
    const C* src = (const C*)in.base + (long long)f * in.fs + ((long long)y * L + j) * in.rs + kx;
    C v[RA];
#pragma unroll
    for (int r = 0; r < RA; ++r) v[r] = ok ? src[(long long)(r * RB) * in.rs] : cmk<C>(0.0, 0.0);
    zpass_a<C, RA, NL, false>(v, buf, li, j);
  }
  __syncthreads();
  const long long kzs = (long long)Kx * out.ps;
  for (int t = threadIdx.x; t < NL * RA; t += NT) {
    const int li = t % NL, k = t / NL;
    C v[RB];
    zpass_b<C, RA, RB, NL, false>(v, buf, tw, li, k);
    const int kx = kx0 + li / TY, y = y0 + li % TY;
    if (kx < Kx && y < Py) {
      C* dst = field_base<C>(out, f) + (long long)kx * out.ps + y + (long long)k * kzs;
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        const int n = k + r * RA;  // kept: n <= Nz/2 and n > L - Nz/2
        if (r * RA <= hz) {
          if (n <= hz) dst[(long long)(r * RA) * kzs] = v[r];
        }
        if (r * RA + RA - 1 > L - Nz + hz) {
          if (n > L - Nz + hz) dst[(long long)(r * RA - (L - Nz)) * kzs] = v[r];
        }
      }
    }
  }
}

// Tiles of the two-pass forms, measured at 384 x 384 x 512
// (inverse / forward, us): FP64 4 x 2 lines on 128 threads, three CTAs per SM
// 466 / 240, four CTAs (no registers to keep a radix-24 butterfly's loads in
// flight) 511 / 246, 4 x 4 lines on 256 threads 476 / 246; at 192 x 192 x 256
// 4 x 4 lines on 128 threads 64 / 36, 4 x 2 on 64 96 / 50, 8 x 2 71 / 34; at
// 256 x 256 x 256 4 x 2 lines, four CTAs 97 / 50, three 98 / 52, 4 x 4 on 128
// threads 104 / 58.
// FP32 at 384: 4 x 4 lines on 256 threads 270 / 130, on 128 288 / 150, 8 x 4
// 293 / 138 (the tensor-staged form, 195 / 115, comes first there).
template <typename C, int L> struct ZTwo {
  enum {
    TX = 4, TY = (sizeof(C) == 8 || L <= 192) ? 4 : 2,
    NT = (sizeof(C) == 8 && L >= 256) ? 256 : 128,
    MB = sizeof(C) == 8 ? 2 : (ZPlan<L>::A <= 18 ? 4 : (ZPlan<L>::A > 24 ? 2 : 3))
  };
};
#define DNS_ZCASE(n) case n: return f(std::integral_constant<int, n>());
template <typename F> cudaError_t with_len_z(int L, F&& f) {
  switch (L) { ZPLAN_LENGTHS(DNS_ZCASE) }
  return cudaErrorNotSupported;
}
template <typename C, class PA>
cudaError_t launch_zb2(PA in, RowArr out, int nf, DnsGeom g, FftTab<C> tab, cudaStream_t st, bool probe) {
  return with_len_z(g.Pz, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    typedef ZTwo<C, L> T;
    if (!tab.zt || g.Nz != L / 3 * 2) return cudaErrorNotSupported;
    if (probe) return cudaSuccess;
    auto k = k_zb2<C, L, T::TX, T::TY, T::NT, T::MB, PA>;
    const size_t sm = (size_t)L * T::TX * T::TY * sizeof(C);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<dim3((g.Kx - 1 + T::TX - 1) / T::TX, (g.Py + T::TY - 1) / T::TY, nf), T::NT, sm, st>>>(in, out, g, tab.zt);
    return cudaGetLastError();
  });
}
template <typename C, class PA>
cudaError_t launch_zf2(RowArr in, PA out, int nf, DnsGeom g, FftTab<C> tab, cudaStream_t st, bool probe) {
  return with_len_z(g.Pz, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    typedef ZTwo<C, L> T;
    if (!tab.zt || g.Nz != L / 3 * 2) return cudaErrorNotSupported;
    if (probe) return cudaSuccess;
    auto k = k_zf2<C, L, T::TX, T::TY, T::NT, T::MB, PA>;
    const size_t sm = (size_t)L * T::TX * T::TY * sizeof(C);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<dim3((g.Kx + T::TX - 1) / T::TX, (g.Py + T::TY - 1) / T::TY, nf), T::NT, sm, st>>>(in, out, g, tab.zt);
    return cudaGetLastError();
  });
}
#endif
