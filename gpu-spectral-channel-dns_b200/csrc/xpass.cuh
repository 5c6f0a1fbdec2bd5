// Streamwise (x) pass: half spectra of six fields -> rows of points -> Lamb
// vector with the rotation term -> half spectra of three fields, x 1/(Px Pz).
//
// A CTA of NW warps owns NR rows (pairs of rows share a wall-normal plane).
// Line 3 r + q holds row r's packed pair q, (u, v), (omega_x, omega_y),
// (w, omega_z): two real fields are one complex transform.  A warp takes its
// lines through all inverse passes but the last without a block barrier.  The
// last inverse pass, the Lamb vector and the first forward pass are one: with
// the same radix RF, butterfly k of the last inverse pass ends on the points
// k + m L/RF that butterfly k of the first forward pass starts from, so one
// thread takes the three pairs of its row there, forms the products in
// registers and transforms lambda_x + i lambda_y forward at once (lambda_z of
// the two rows of a pair share a line: the neighbouring lane's values come by
// shuffle).  Lines 3 r then hold lambda_x + i lambda_y of row r, line 6 p + 1
// lambda_z of pair p.
//
// What bounds it: every pass reads and writes each value through shared
// memory at 128 bytes a clock and SM; fusing the middle removes four of the
// transfers of each inverse line (store, Lamb read, write, read).  Measured
// at 384 x 384 x 512 against the form with the Lamb vector between two whole
// transforms: FP32 356 -> 298 us, FP64 987 -> 644; 192 x 192 x 256 FP64
// 125 -> 86; 128 x 128 x 128 FP64, a length without a plan before, 96 -> 29.
#pragma once
#include "kernels.cuh"
#include "wfft.cuh"
#ifdef __CUDACC__
#include "mbar.cuh"
#endif

// RF and the other radices (inverse: PRE..., RF; forward: RF, PRE...), rows
// per CTA and warps.  A row pair's 2 L/RF butterflies fit the CTA's threads;
// three pairs of RF complex values stay in registers (RF <= 18 FP32, 9 FP64).
// Chosen by measurement where that leaves a choice (us; FP64 with 256 points along
// the wall normal, 192: 8 with 24 86, with 6, 4 105; 216: 9 with 24 134, with 6, 4
// 158; 144: 8 with 18 61, 9 with 16 73; FP32 96: 8 with 12 95, 4 with 24 115; 128:
// eight rows 60, four 64).
template <int L, int MAXR> struct XPlan { enum { ok = 0 }; };
#define XPLAN(L, MAXR, RF_, NR_, NW_, ...)                                \
  template <> struct XPlan<L, MAXR> {                                     \
    enum { ok = 1, RF = RF_, NR = NR_, NW = NW_ };                        \
    typedef Radices<__VA_ARGS__> PRE;                                     \
    typedef Radices<__VA_ARGS__, RF_> INV;                                \
    typedef Radices<RF_, __VA_ARGS__> FWD;                                \
  };
// FP32
XPLAN(24, 16, 4, 8, 3, 6)
XPLAN(32, 16, 4, 8, 3, 8)
XPLAN(36, 16, 6, 8, 3, 6)
XPLAN(48, 16, 4, 8, 3, 12)
XPLAN(54, 16, 6, 8, 3, 9)
XPLAN(64, 16, 8, 8, 3, 8)
XPLAN(72, 16, 4, 8, 3, 18)
XPLAN(96, 16, 8, 8, 3, 12)
XPLAN(108, 16, 6, 8, 3, 18)
XPLAN(128, 16, 8, 8, 3, 16)
XPLAN(144, 16, 6, 4, 3, 24)
XPLAN(162, 16, 9, 4, 3, 18)
XPLAN(192, 16, 8, 4, 3, 24)
XPLAN(216, 16, 9, 4, 3, 24)
XPLAN(256, 16, 16, 4, 3, 16)
XPLAN(288, 16, 12, 4, 3, 24)
XPLAN(324, 16, 18, 4, 3, 18)
XPLAN(384, 16, 16, 4, 3, 24)
XPLAN(432, 16, 18, 4, 3, 24)
XPLAN(512, 16, 16, 4, 3, 32)
XPLAN(576, 16, 16, 4, 3, 6, 6)
XPLAN(768, 16, 16, 4, 3, 8, 6)
// FP64
XPLAN(24, 8, 4, 8, 3, 6)
XPLAN(32, 8, 4, 8, 3, 8)
XPLAN(36, 8, 6, 8, 3, 6)
XPLAN(48, 8, 4, 8, 3, 12)
XPLAN(54, 8, 6, 8, 3, 9)
XPLAN(64, 8, 8, 8, 3, 8)
XPLAN(72, 8, 6, 8, 3, 12)
XPLAN(96, 8, 8, 8, 3, 12)
XPLAN(108, 8, 9, 8, 3, 12)
XPLAN(128, 8, 8, 4, 3, 16)
XPLAN(144, 8, 8, 4, 3, 18)
XPLAN(162, 8, 9, 4, 3, 18)
XPLAN(192, 8, 8, 4, 3, 24)
XPLAN(216, 8, 9, 4, 3, 24)
XPLAN(256, 8, 8, 2, 3, 8, 4)
XPLAN(288, 8, 9, 2, 3, 8, 4)
XPLAN(324, 8, 9, 2, 3, 6, 6)
XPLAN(384, 8, 8, 2, 3, 8, 6)
XPLAN(432, 8, 9, 2, 3, 8, 6)
XPLAN(512, 8, 8, 4, 6, 8, 8)
XPLAN(576, 8, 9, 4, 6, 8, 8)
XPLAN(768, 8, 8, 4, 6, 12, 8)
#undef XPLAN
#define XPLAN_LENGTHS(X) \
  X(24) X(32) X(36) X(48) X(54) X(64) X(72) X(96) X(108) X(128) X(144) X(162) X(192) X(216) X(256) X(288) \
  X(324) X(384) X(432) X(512) X(576) X(768)

// Twiddles: the inverse plan's passes, then the forward plan's, every value
// rounded from W, the table W_L^j, j < L.  FP64 products w, w^2, w^3, ... would
// save loads, but their error grows with the radix: rms error of a forward line
// (1e-16) 4.6 by products and 1.8 from the table at 192, 5.1 and 2.0 at 216, 3.0
// and 1.9 at 384; 384 x 384 x 512 634 -> 644 us, 192 x 192 x 256 84 -> 86.
template <typename C, int... Rs> void xtw_fill(Radices<Rs...>, int L, const double2* W, C* out) {
  const int rs[] = {Rs...};
  int ns = 1;
  for (int i = 0; i < (int)sizeof...(Rs); ++i) {
    const int R = rs[i];
    if (ns > 1)
      for (int r = 1; r < R; ++r)
        for (int k = 0; k < ns; ++k) *out++ = from_d2<C>(W[r * k * (L / (ns * R))]);
    ns *= R;
  }
}
template <typename C> int xtw_table(int L, const double2* W, std::vector<C>& out) {
  switch (L) {
#define XCASE(n)                                                    \
  case n: {                                                         \
    typedef XPlan<n, FftMaxRadix<C>::v> P;                          \
    const int ni = wtw_size(typename P::INV()), nf = wtw_size(typename P::FWD()); \
    out.resize((size_t)(ni + nf));                                  \
    xtw_fill(typename P::INV(), n, W, out.data());                  \
    xtw_fill(typename P::FWD(), n, W, out.data() + ni);             \
    return ni + nf;                                                 \
  }
    XPLAN_LENGTHS(XCASE)
#undef XCASE
  }
  return -1;
}

// One butterfly of a pass (radix R, Ns = product of the earlier radices) on
// a padded line (positions wsw(i)); TWO: the pass's twiddles in the table
template <typename C, int L, int R, int Ns, int TWO, bool INV> struct XPass {
  static constexpr int NB = L / R, S = WSwz<C>::S, M = (1 << S) - 1;
  static_assert(L % R == 0, "radix does not divide the length");
  static constexpr bool LIN_LD = (NB & M) == 0;
  static constexpr bool LIN_ST = wlin_store(M, NB, Ns, R);
  DNS_HD static void load(const C* x, int j, C* v) {
    if constexpr (LIN_LD) {
      const C* xb = x + wsw<C>(j);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = xb[wsw<C>(r * NB)];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = x[wsw<C>(j + r * NB)];
    }
  }
  // the twiddles w[1..R-1] of butterfly j
  DNS_HD static void weights(const C* tw, int j, C* w) {
    const int k = j % Ns;
#pragma unroll
    for (int r = 1; r < R; ++r) w[r] = tw[TWO + (r - 1) * Ns + k];
  }
  DNS_HD static void run(C* v, const C* w) {
    if constexpr (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = INV ? cmulc(v[r], w[r]) : cmul(v[r], w[r]);
    }
    Codelet<R, INV, C>::run(v);
  }
  DNS_HD static int out(int j) { return (j / Ns) * Ns * R + j % Ns; }  // outputs out(j) + r Ns
  DNS_HD static void store(C* y, int j, const C* v) {
    if constexpr (LIN_ST) {
      C* yb = y + wsw<C>(out(j));
#pragma unroll
      for (int r = 0; r < R; ++r) yb[wsw<C>(r * Ns)] = v[r];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) y[wsw<C>(out(j) + r * Ns)] = v[r];
    }
  }
};

#ifdef __CUDACC__
// The passes of a radix list by one warp on NL lines, line l at at(l); the
// first pass (Ns = 1) reads element n of line l from ld(l, n); STOP leaves the
// last radix of the list to the caller; keep(k): whether output k of the last
// pass is stored.
template <typename C, int L, int NL, bool INV, int Ns, int TWO, bool LD, int STOP, int R, int... Rest> struct XRun {
  template <class AT, class LDF, class KEEP>
  __device__ __forceinline__ static void go(const C* tw, int lane, AT at, LDF ld, KEEP keep) {
    if constexpr ((int)sizeof...(Rest) >= STOP) {
      typedef XPass<C, L, R, Ns, TWO, INV> P;
      constexpr int NT = NL * P::NB, B = (NT + 31) / 32;
      C v[B][R];
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int i = lane + 32 * q;
        if (NT % 32 && i >= NT) continue;
        const int l = i / P::NB, j = i - l * P::NB;
        WFFT_ASSUME(j >= 0 && j < P::NB);
        if constexpr (LD) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[q][r] = ld(l, j + r * P::NB);
          P::run(v[q], nullptr);
        } else {
          C w[R];
          if constexpr (Ns > 1) P::weights(tw, j, w);
          P::load(at(l), j, v[q]);
          P::run(v[q], w);
        }
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int i = lane + 32 * q;
        if (NT % 32 && i >= NT) continue;
        const int l = i / P::NB, j = i - l * P::NB;
        WFFT_ASSUME(j >= 0 && j < P::NB);
        if constexpr (sizeof...(Rest) == 0) {
          C* y = at(l);
          const int b = P::out(j);
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (keep(b + r * Ns)) y[wsw<C>(b + r * Ns)] = v[q][r];
        } else {
          P::store(at(l), j, v[q]);
        }
      }
      __syncwarp();
      if constexpr (sizeof...(Rest) > 0)
        XRun<C, L, NL, INV, Ns * R, TWO + (Ns > 1 ? (R - 1) * Ns : 0), false, STOP, Rest...>::go(tw, lane, at, ld, keep);
    }
  }
};
template <typename C, int L, int NL, bool INV, int Ns, int TWO, bool LD, int STOP, class RS> struct XDo;
template <typename C, int L, int NL, bool INV, int Ns, int TWO, bool LD, int STOP, int... Rs>
struct XDo<C, L, NL, INV, Ns, TWO, LD, STOP, Radices<Rs...>>
    : XRun<C, L, NL, INV, Ns, TWO, LD, STOP, Rs...> {};

// line stride: the two rows of a pair fall half the banks apart
template <typename C> constexpr int xline(int L) {
  const int per = 128 / (int)sizeof(C), half = per / 2;
  int n = wlen<C>(L);
  while (n % per != half) ++n;
  return n;
}
// lines a warp takes through the inverse passes at once: at most 24 complex
// values a lane
constexpr int xbatch(int L, int lines) {
  int n = lines;
  while (n > 1 && (n * L > 24 * 32 || lines % n)) --n;
  return n;
}

// SC: row groups of the plan per CTA (its rows and warps times SC)
template <typename C, int L, int SC, int MB>
__global__ void __launch_bounds__(32 * SC * XPlan<L, FftMaxRadix<C>::v>::NW, MB)
    k_x2(RowArr in, RowArr out, DnsGeom g, const C* __restrict__ tw, const double* __restrict__ Uy, double Ro,
         const double* __restrict__ runs, int* status) {
  typedef XPlan<L, FftMaxRadix<C>::v> P;
  typedef T_of<C> T;
  constexpr int NR = SC * P::NR, NW = SC * P::NW, RF = P::RF, NB = L / RF, LW = xline<C>(L), NT = 32 * NW;
  constexpr int LPW = 3 * NR / NW;                          // inverse lines per warp
  constexpr int NF = 3 * NR / 2, FPW = (NF + NW - 1) / NW;  // forward lines, per warp
  constexpr int hx = L / 3;                                 // Nx / 2 (the launcher checks it)
  constexpr int SR = (hx + 7) / 8 * 8;                      // staged bins of a half spectrum
  static_assert(3 * NR % NW == 0 && 2 * NB <= NT && 2 * SR <= LW, "plan");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t bars[NW];
  C* z = (C*)smem_raw;  // 3 NR lines
  const unsigned nrows = (unsigned)((long long)g.Py * g.Pz * g.nrun);  // a batch: members' rows one after another
  const unsigned r0 = blockIdx.x * NR;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  C* zw = z + (size_t)(LPW * warp) * LW;
  // this warp's half spectra (bins 0..Nx/2-1), two in each of its lines: the
  // first pass of a batch of lines reads them before it writes the lines
  uint64_t* bar = bars + warp;
  if (lane == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
    mbar_expect_tx(bar, 2 * LPW * SR * sizeof(C));
  }
  __syncwarp();
  for (int i = lane; i < 2 * LPW; i += 32) {
    const int line = LPW * warp + (i >> 1);
    const int rl = line / 3, q = line - 3 * rl;
    const unsigned row = min(r0 + rl, nrows - 1);  // beyond the last row: duplicate work, not stored
    // fields of similar magnitude share a transform: (u, v), (ox, oy), (w, oz)
    const int fa = q == 0 ? 0 : (q == 1 ? 3 : 2), fb = q == 0 ? 1 : (q == 1 ? 4 : 5);
    bulk_g2s(zw + (size_t)(i >> 1) * LW + (i & 1) * SR,
             (const C*)in.base + (long long)((i & 1) ? fb : fa) * in.fs + (long long)row * in.rs, SR * sizeof(C), bar);
  }
  // a wait that runs out is reported and waited once more (bounded); the
  // warp then goes on, so that every warp reaches the block barriers
  if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar, 0, 1LL << 31, status))) {
    if (lane == 0) {
      atomicOr(status, 1);
      mbar_wait_bounded(bar, 0, 1LL << 31, nullptr);
    }
    __syncwarp();
  }
  constexpr int NLB = xbatch(L, LPW);
#pragma unroll 1
  for (int b = 0; b < LPW; b += NLB) {
    C* zb = zw + (size_t)b * LW;
    auto at = [&](int l) { return zb + l * LW; };
    // Z = A + iB over the full length: IFFT(Z) = a(x) + i b(x); the
    // imaginary parts of the DC bins are dropped (C2R convention), Nyquist
    // and padding are zero
    auto ld = [&](int l, int n) -> C {
      const C* a = zb + l * LW;
      const C* bb = a + SR;
      if (n == 0) { C r; r.x = a[0].x; r.y = bb[0].x; return r; }
      if (n < hx) {
        const C av = a[n], bv = bb[n];
        C r; r.x = av.x - bv.y; r.y = av.y + bv.x; return r;
      }
      if (n > L - hx) {  // conj(a) + i conj(b)
        const C av = a[L - n], bv = bb[L - n];
        C r; r.x = av.x + bv.y; r.y = bv.x - av.y; return r;
      }
      return cmk<C>(0.0, 0.0);
    };
    XDo<C, L, NLB, true, 1, 0, true, 1, typename P::INV>::go(tw, lane, at, ld, [](int) { return true; });
  }
  __syncthreads();
  // last inverse pass, Lamb vector, first forward pass: PPR row pairs a
  // round, thread t: row t & 1 of the pair, butterfly k
  constexpr int PPR = NT / (2 * NB) < NR / 2 ? NT / (2 * NB) : NR / 2;
  constexpr int TWI = wtw_offset(typename P::INV(), L / RF);
  typedef XPass<C, L, RF, L / RF, TWI, true> PI;
  typedef XPass<C, L, RF, 1, 0, false> PF;
  const unsigned pr = (unsigned)(g.Py * g.Pz);
#pragma unroll 1
  for (int p0 = 0; p0 < NR / 2; p0 += PPR) {
    const int t = threadIdx.x, pi = t / (2 * NB);
    const bool act = pi < PPR && p0 + pi < NR / 2;
    const int p = act ? p0 + pi : p0, k = act ? (t - pi * 2 * NB) >> 1 : 0, row = 2 * p + (t & 1);
    // both rows of a pair lie in one wall-normal plane of one member
    const unsigned gr = min(r0 + 2 * p, nrows - 1);
    const unsigned run = gr / pr, y = (gr - run * pr) / (unsigned)g.Pz;
    const T ro = (T)(runs ? runs[3 * run + 1] : Ro), Ub = (T)Uy[y];
    C* zr = z + (size_t)(3 * row) * LW;
    C f[3][RF];
    {
      C w[RF];
      PI::weights(tw, k, w);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        PI::load(zr + q * LW, k, f[q]);
        PI::run(f[q], w);
      }
    }
    // f[0] <- lambda_x + i lambda_y; f[1].x <- lambda_z
#pragma unroll
    for (int r = 0; r < RF; ++r) {
      const T u = f[0][r].x, v = f[0][r].y, ox = f[1][r].x, oy = f[1][r].y, w = f[2][r].x, oz = f[2][r].y;
      f[0][r].x = oz * v - oy * w - ro * w;
      f[0][r].y = ox * w - oz * u;
      f[1][r].x = oy * u - ox * v + ro * (u + Ub);
    }
#pragma unroll
    for (int r = 0; r < RF; ++r) f[1][r].y = __shfl_down_sync(0xffffffffu, f[1][r].x, 1);
    PF::run(f[0], nullptr);
    __syncthreads();  // every read of the round's lines is done
    if (act) {
      PF::store(zr, k, f[0]);
      if (!(t & 1)) {
        PF::run(f[1], nullptr);
        PF::store(zr + LW, k, f[1]);
      }
    }
  }
  __syncthreads();
  // the other forward passes: line f < NR is lambda_x + i lambda_y of row f
  // (z line 3 f), line NR + p lambda_z of pair p (z line 6 p + 1); only the
  // bins the half spectra need are stored
  const int Kx = g.Kx;
  if (FPW * warp < NF) {
    auto at = [&](int l) {
      const int f = FPW * warp + l;
      return z + (size_t)(f < NR ? 3 * f : 6 * (f - NR) + 1) * LW;
    };
    constexpr int NLF = xbatch(L, FPW);
#pragma unroll 1
    for (int b = 0; b < FPW; b += NLF) {
      auto atb = [&](int l) { return at(b + l); };
      const C* twf = tw + wtw_size(typename P::INV());
      XDo<C, L, NLF, false, RF, 0, false, 0, typename P::PRE>::go(
          twf, lane, atb, 0, [](int kk) { return kk <= hx || kk >= L - hx; });
    }
  }
  __syncthreads();
  // unpack: output row o = 3 rl + fl (field fl of row rl), lanes over the
  // bins k; shared loads of a batch before its stores
  const T sc = (T)(0.5 / ((double)g.Px * (double)g.Pz));
  constexpr int KB = (hx + 1 + 31) / 32, XB = KB < 5 ? KB : 5;
  for (int o = warp; o < 3 * NR; o += NW) {
    const int rl = o / 3, fl = o - 3 * rl;
    if (r0 + rl >= nrows) break;
    const C* Z = z + (size_t)(fl < 2 ? 3 * rl : 6 * (rl >> 1) + 1) * LW;
    const bool im = (fl < 2) ? (fl == 1) : (rl & 1);
    C* dst = (C*)out.base + (long long)fl * out.fs + (long long)(r0 + rl) * out.rs;
    for (int k0 = lane; k0 < Kx; k0 += 32 * XB) {
      C zk[XB], zm[XB];
#pragma unroll
      for (int u = 0; u < XB; ++u) {
        const int k = min(k0 + 32 * u, hx);
        zk[u] = Z[wsw<C>(k)];
        zm[u] = Z[wsw<C>(k ? L - k : 0)];
      }
#pragma unroll
      for (int u = 0; u < XB; ++u) {
        const int k = k0 + 32 * u;
        if (k >= Kx) continue;
        C v;
        if (!im) { v.x = zk[u].x + zm[u].x; v.y = zk[u].y - zm[u].y; }
        else { v.x = zk[u].y + zm[u].y; v.y = zm[u].x - zk[u].x; }
        dst[k] = v * sc;
      }
    }
  }
}
#endif
