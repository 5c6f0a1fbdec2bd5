// The time step's spanwise (z) and streamwise (x) passes.
//
// Reference counterparts:
//   transpose_forward / transpose_backward ... source/transpose.cu:223-257, 358-382
//   setZerosKernel ........................... source/transform.cu:355-377
//   2D cuFFT Z2D / D2Z + normalizeKernel ..... source/transform.cu:176, 240, 388-412
//   computeLambVectorKernel / computeLambDevice source/nonlinear.cu:366-428
//
// Spanwise pass: a CTA owns a tile of TX streamwise modes x TY wall-normal
// points and transforms those TX*TY lines along the span in shared memory.
// It reads one layout (pencil-major, wall-normal index contiguous) and
// writes the other (row-major, streamwise index contiguous) with TX- or
// TY-element contiguous runs, so the x-y-z transpose, the span remap
// ky' = ky or ky + Pz - Nz, the zero padding Nz -> Pz (and truncation), and
// the zeroing of both Nyquist modes are folded into the one pass.
//
// Streamwise pass: two real rows share one complex FFT (a + i b).
//
// zxstep_f64.cu and zxstep_f32.cu instantiate a precision each (the reason stands
// in ystep.cuh).
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include <type_traits>

#include "fftline.cuh"
#include "kernels.cuh"
#include "mbar.cuh"
#include "xpass.cuh"
#include "zpass.cuh"
#include "zxline.cuh"
#include "zxpass.cuh"

// ---------------------------------------------------------------------------
// spanwise backward: pencils [f][kz*Kx+kx][y] -> rows [f][y][zp][kx]
// ---------------------------------------------------------------------------
template <typename C, int TX, int TY, int L>
__global__ void __launch_bounds__(256, 3) k_zb(PencilArr in, RowArr out, DnsGeom g, FftTab<C> tab) {
  typedef FLine<C, L> FL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* lines = (C*)smem_raw;
  const int Pz = L > 0 ? L : g.Pz;
  const int Nz = g.Nz, Kx = g.Kx, Py = g.Py;
  const int ls = FL::stride(Pz);
  const int kx0 = blockIdx.x * TX;
  const int y0 = blockIdx.y * TY;
  const int f = blockIdx.z;
  const int NL = TX * TY;
  const int hz = Nz / 2;
  // zero band [Nz/2, Pz - Nz/2] (Nyquist and padding)
  const int nzero = Pz - Nz + 1;
  for (int t = threadIdx.x; t < NL * nzero; t += blockDim.x) {
    const int li = t / nzero;
    const int n = hz + (t - li * nzero);
    lines[(size_t)li * ls + FL::in_pos(tab, n)] = cmk<C>(0.0, 0.0);
  }
  for (int t = threadIdx.x; t < Nz * NL; t += blockDim.x) {
    const int yl = t % TY;
    const int kxl = (t / TY) % TX;
    const int kz = t / NL;
    if (kz == hz) continue;
    const int n = (kz < hz) ? kz : kz + (Pz - Nz);
    const int kx = kx0 + kxl;
    const int y = y0 + yl;
    C v = cmk<C>(0.0, 0.0);
    if (kx < Kx - 1 && y < Py) v = ppen<C>(in, f, (long long)kz * Kx + kx)[y];
    lines[(size_t)(kxl * TY + yl) * ls + FL::in_pos(tab, n)] = v;
  }
  FL::template fft<true>(lines, NL, ls, tab);
  for (int t = threadIdx.x; t < TY * Pz * TX; t += blockDim.x) {
    const int kxl = t % TX;
    const int zp = (t / TX) % Pz;
    const int yl = t / (TX * Pz);
    const int kx = kx0 + kxl;
    const int y = y0 + yl;
    if (kx < Kx && y < Py)
      prow<C>(out, f, (long long)y * Pz + zp)[kx] = lines[(size_t)(kxl * TY + yl) * ls + FL::out_pos(zp)];
  }
}

// ---------------------------------------------------------------------------
// spanwise forward: rows [f][y][zp][kx] -> pencils [f][kz*Kx+kx][y]
// ---------------------------------------------------------------------------
template <typename C, int TX, int TY, int L>
__global__ void __launch_bounds__(256, 3) k_zf(RowArr in, PencilArr out, DnsGeom g, FftTab<C> tab) {
  typedef FLine<C, L> FL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* lines = (C*)smem_raw;
  const int Pz = L > 0 ? L : g.Pz;
  const int Nz = g.Nz, Kx = g.Kx, Py = g.Py;
  const int ls = FL::stride(Pz);
  const int kx0 = blockIdx.x * TX;
  const int y0 = blockIdx.y * TY;
  const int f = blockIdx.z;
  const int NL = TX * TY;
  for (int t = threadIdx.x; t < TY * Pz * TX; t += blockDim.x) {
    const int kxl = t % TX;
    const int zp = (t / TX) % Pz;
    const int yl = t / (TX * Pz);
    const int kx = kx0 + kxl;
    const int y = y0 + yl;
    C v = cmk<C>(0.0, 0.0);
    if (kx < Kx && y < Py) v = prow<C>(in, f, (long long)y * Pz + zp)[kx];
    lines[(size_t)(kxl * TY + yl) * ls + FL::in_pos(tab, zp)] = v;
  }
  FL::template fft<false>(lines, NL, ls, tab);
  const int hz = Nz / 2;
  for (int t = threadIdx.x; t < Nz * NL; t += blockDim.x) {
    const int yl = t % TY;
    const int kxl = (t / TY) % TX;
    const int kz = t / NL;
    const int kx = kx0 + kxl;
    const int y = y0 + yl;
    const int n = (kz <= hz) ? kz : kz + (Pz - Nz);
    if (kx < Kx && y < Py)
      ppen<C>(out, f, (long long)kz * Kx + kx)[y] = lines[(size_t)(kxl * TY + yl) * ls + FL::out_pos(n)];
  }
}

// Same spanwise passes in FP32 on tensor-staged tiles of 16 lines (streamwise
// modes x wall-normal points), eight warps with a pair of lines each: a warp
// loads its pair by tiled 4-D copies into its own part of shared memory (the
// box's innermost extent is the pair, 16 bytes), takes pass A of the plan from
// there (every input is read before an output is stored) and pass B, shared by
// the CTA, stores the lines straight to global memory.  Element pos of line l
// of a pair sits at 2 (pos + pos / RA) + l: the lanes of pass A, RA apart, and
// those of pass B, which take the 16 lines of a position (pairs WS apart), fall
// in distinct banks.  384 x 384 x 512, inverse / forward: 195 / 115 us, against
// 230 / 124 with both passes by the warp and the tile's rows or pencils written
// from shared memory in a third.  The tile: ZStage (zpass.cuh).
namespace {
template <typename C, int L, bool INV, class LD>
__device__ __forceinline__ void zstage_a(C* wl, int lane, LD ld) {
  typedef ZStage<C, L> Z;
  C v[Z::RA];
  const int l = lane & 1, j = lane >> 1;
  if (j < Z::RB) {
    WFFT_ASSUME(j >= 0 && j < Z::RB);
#pragma unroll
    for (int r = 0; r < Z::RA; ++r) v[r] = ld(l, j + r * Z::RB);
    Codelet<Z::RA, INV, C>::run(v);
  }
  __syncwarp();
  if (j < Z::RB) {
    C* o = wl + 2 * j * (Z::RA + 1) + l;
#pragma unroll
    for (int r = 0; r < Z::RA; ++r) o[2 * r] = v[r];
  }
}
template <typename C, int L, bool INV>
__device__ __forceinline__ void zstage_b(C* v, const C* line, const C* __restrict__ tw, int k) {
  typedef ZStage<C, L> Z;
#pragma unroll
  for (int r = 0; r < Z::RB; ++r) v[r] = line[2 * (k + r * (Z::RA + 1))];
#pragma unroll
  for (int r = 1; r < Z::RB; ++r) {
    const C w = tw[(r - 1) * Z::RA + k];
    v[r] = INV ? cmulc(v[r], w) : cmul(v[r], w);
  }
  Codelet<Z::RB, INV, C>::run(v);
}
// a wait that runs out is reported and waited once more (bounded); the warp
// then goes on, so that every warp reaches the block barriers
__device__ __forceinline__ void zstage_wait(uint64_t* bar, int lane, int* status) {
  if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar, 0, 1LL << 31, status))) {
    if (lane == 0) {
      atomicOr(status, 1);
      mbar_wait_bounded(bar, 0, 1LL << 31, nullptr);
    }
    __syncwarp();
  }
}
}  // namespace

// Inverse pass, 8 x 2 tile (64-byte runs on the row side): warp w owns kx0 + w
// and two consecutive y (box y 2 x kx 1 x kz Nz x field 1, 4 KB at Nz = 256).
// Rows beyond Py read as the copy's zero fill; the streamwise Nyquist column
// (kx = Kx - 1) is zero and not read later: it is left out.
template <typename C, int L>
__global__ void __launch_bounds__(256, 3) k_zbt(const __grid_constant__ CUtensorMap tin, RowArr out,
                                                DnsGeom g, const C* __restrict__ tw, int* status) {
  typedef ZStage<C, L> Z;
  constexpr int Nz = L / 3 * 2, hz = Nz / 2;  // my / 3 * 2 (the launcher checks g.Nz)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t bars[8];
  C* lines = (C*)smem_raw;
  const int kx0 = blockIdx.x * 8, y0 = blockIdx.y * 2, f = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  C* wl = lines + (size_t)warp * Z::WS;
  const C* tile = (const C*)(((uintptr_t)wl + 127) & ~(uintptr_t)127);  // [kz][y pair]
  if (lane == 0) {
    mbar_init(bars + warp, 1);
    fence_mbar_init();
    mbar_expect_tx(bars + warp, (uint32_t)(2 * Nz * sizeof(C)));
    tma_load_4d((void*)tile, &tin, y0, kx0 + warp, 0, f, bars + warp);
  }
  __syncwarp();
  zstage_wait(bars + warp, lane, status);
  zstage_a<C, L, true>(wl, lane, [&](int l, int n) -> C {
    if (n < hz) return tile[2 * n + l];
    if (n > L - hz) return tile[2 * (n - (L - Nz)) + l];
    return cmk<C>(0.0, 0.0);
  });
  __syncthreads();
  for (int t = threadIdx.x; t < 16 * Z::RA; t += 256) {
    const int kxl = t & 7, yl = (t >> 3) & 1, k = t >> 4;
    const int kx = kx0 + kxl, y = y0 + yl;
    C v[Z::RB];
    zstage_b<C, L, true>(v, lines + (size_t)kxl * Z::WS + yl, tw, k);
    if (kx < g.Kx - 1 && y < g.Py) {
      C* dst = prow<C>(out, f, (long long)y * L + k) + kx;
#pragma unroll
      for (int r = 0; r < Z::RB; ++r) dst[(long long)(r * Z::RA) * out.rs] = v[r];
    }
  }
}

// Forward pass, 4 x 4 tile (32-byte runs on the pencil side): warp w owns y0 +
// w / 2 and a kx pair, one copy of the whole line up to 256 points, two of its
// halves beyond (box kx 2 x zp ROWS x y 1 x field 1).  Rows beyond Py and columns
// beyond Kx read as the copy's zero fill.
template <typename C, int L>
__global__ void __launch_bounds__(256, 3) k_zft(const __grid_constant__ CUtensorMap tin, PencilArr out,
                                                DnsGeom g, const C* __restrict__ tw, int* status) {
  typedef ZStage<C, L> Z;
  static_assert(Z::copies_ok, "a copy's destination is 128-byte aligned");
  constexpr int Nz = L / 3 * 2, hz = Nz / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint64_t bars[8];
  C* lines = (C*)smem_raw;
  const int Kx = g.Kx, Py = g.Py;
  const int kx0 = blockIdx.x * 4, y0 = blockIdx.y * 4, f = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  C* wl = lines + (size_t)warp * Z::WS;
  C* tile = (C*)(((uintptr_t)wl + 127) & ~(uintptr_t)127);  // [zp][kx pair]
  if (lane == 0) {
    mbar_init(bars + warp, 1);
    fence_mbar_init();
    mbar_expect_tx(bars + warp, (uint32_t)(2 * L * sizeof(C)));
    const int x = kx0 + 2 * (warp & 1), y = y0 + (warp >> 1);
#pragma unroll
    for (int z = 0; z < L; z += Z::ROWS) tma_load_4d(tile + 2 * z, &tin, x, z, y, f, bars + warp);
  }
  __syncwarp();
  zstage_wait(bars + warp, lane, status);
  zstage_a<C, L, false>(wl, lane, [&](int l, int n) -> C { return tile[2 * n + l]; });
  __syncthreads();
  const long long kzs = (long long)Kx * out.ps;
  for (int t = threadIdx.x; t < 16 * Z::RA; t += 256) {
    const int yl = t & 3, kxl = (t >> 2) & 3, k = t >> 4;
    const int kx = kx0 + kxl, y = y0 + yl;
    C v[Z::RB];
    zstage_b<C, L, false>(v, lines + (size_t)(2 * yl + (kxl >> 1)) * Z::WS + (kxl & 1), tw, k);
    if (kx < Kx && y < Py) {
      C* dst = ppen<C>(out, f, kx) + y + (long long)k * kzs;
#pragma unroll
      for (int r = 0; r < Z::RB; ++r) {
        const int n = k + r * Z::RA;  // kept: n <= Nz/2 and n > L - Nz/2
        if (r * Z::RA <= hz) {
          if (n <= hz) dst[(long long)(r * Z::RA) * kzs] = v[r];
        }
        if (r * Z::RA + Z::RA - 1 > L - Nz + hz) {
          if (n > L - Nz + hz) dst[(long long)(r * Z::RA - (L - Nz)) * kzs] = v[r];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// fused streamwise pass: 6 half-spectra rows -> physical -> Lamb vector with
// the rotation term -> 3 half-spectra rows, x 1/(Px Pz).
// Input fields u, v(span), w(wall), omega_x, omega_y, omega_z; output
// lambda_x, lambda_y(span), lambda_z(wall).  Two rows per CTA.
// ---------------------------------------------------------------------------
template <typename C, int L>
__global__ void __launch_bounds__(256, 3) k_x_fused(RowArr in, RowArr out, DnsGeom g, FftTab<C> tab,
                                                   const double* __restrict__ Uy, double Ro,
                                                   const double* __restrict__ runs) {
  // two rows per CTA: lines 0-2 hold row 0's packed fields (u,v) (ox,oy)
  // (w,oz), lines 3-5 row 1's; after the inverse transform a thread owning
  // point j of both rows writes lambda_x + i lambda_y of row 0 / row 1 into
  // lines 0 / 1 and lambda_z(row 0) + i lambda_z(row 1) into line 2 at the
  // same position, then lines 0-2 are transformed forward.
  typedef FLine<C, L> FL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef T_of<C> T;
  const int Px = L > 0 ? L : g.Px;
  const int hx = g.Nx / 2;
  const int ls = FL::stride(Px);
  C* z = (C*)smem_raw;  // 6 lines (9 for the runtime-length FFT)
  // a batch: members' rows one after another, pairs within a member
  const long long pr = (long long)g.Py * g.Pz, np = (pr + 1) / 2;
  const int run = (int)(blockIdx.x / np);
  const long long r0 = run * pr + 2 * (blockIdx.x - run * np), nrows = (run + 1) * pr;
  for (int t = threadIdx.x; t < 2 * 3 * Px; t += blockDim.x) {
    const int rl = t / (3 * Px);
    const int rem = t - rl * 3 * Px;
    const int q = rem / Px;
    const int n = rem - q * Px;
    const long long row = r0 + rl;
    C zz = cmk<C>(0.0, 0.0);
    if (row < nrows) {
      // fields of similar magnitude share a transform (the smaller one's
      // rounding error is relative to the larger): (u, v), (ox, oy), (w, oz)
      const int fa = (q == 0) ? 0 : (q == 1 ? 3 : 2);
      const int fb = (q == 0) ? 1 : (q == 1 ? 4 : 5);
      zz = pack_c2r<C>(prow<C>(in, fa, row), prow<C>(in, fb, row), n, Px, hx);
    }
    z[(size_t)(rl * 3 + q) * ls + FL::in_pos(tab, n)] = zz;
  }
  FL::template fft<true>(z, 6, ls, tab);
  const T ro = (T)(runs ? runs[3 * run + 1] : Ro);
  T Ub[2];  // of each row's plane: with an odd number of rows a plane the two may differ
#pragma unroll
  for (int rl = 0; rl < 2; ++rl) Ub[rl] = (T)Uy[(int)((min(r0 + rl, nrows - 1) - run * pr) / g.Pz)];
  for (int j = threadIdx.x; j < Px; j += blockDim.x) {
    const int op = FL::out_pos(j);
    T lz[2];
    C A[2];
#pragma unroll
    for (int rl = 0; rl < 2; ++rl) {
      const C z0 = z[(size_t)(rl * 3 + 0) * ls + op];
      const C z1 = z[(size_t)(rl * 3 + 1) * ls + op];
      const C z2 = z[(size_t)(rl * 3 + 2) * ls + op];
      const T u = z0.x, v = z0.y, ox = z1.x, oy = z1.y, w = z2.x, oz = z2.y;
      A[rl].x = oz * v - oy * w - ro * w;
      A[rl].y = ox * w - oz * u;
      lz[rl] = oy * u - ox * v + ro * (u + Ub[rl]);
    }
    if (L > 0) {  // natural order: write in place
      z[(size_t)0 * ls + op] = A[0];
      z[(size_t)1 * ls + op] = A[1];
      C B; B.x = lz[0]; B.y = lz[1];
      z[(size_t)2 * ls + op] = B;
    } else {      // digit-reversed input order: separate lines 6-8
      const int pos = FL::in_pos(tab, j);
      z[(size_t)6 * ls + pos] = A[0];
      z[(size_t)7 * ls + pos] = A[1];
      C B; B.x = lz[0]; B.y = lz[1];
      z[(size_t)8 * ls + pos] = B;
    }
  }
  C* zf = (L > 0) ? z : z + (size_t)6 * ls;
  FL::template fft<false>(zf, 3, ls, tab);
  const int Kx = g.Kx;
  const T sc = (T)(0.5 / ((double)g.Px * (double)g.Pz));
  for (int t = threadIdx.x; t < 2 * 3 * Kx; t += blockDim.x) {
    const int k = t % Kx;
    const int fl = (t / Kx) % 3;
    const int rl = t / (3 * Kx);
    const long long row = r0 + rl;
    if (row >= nrows) continue;
    const C* Z = (fl < 2) ? zf + (size_t)rl * ls : zf + (size_t)2 * ls;
    const bool im = (fl < 2) ? (fl == 1) : (rl == 1);
    const C zk = Z[FL::out_pos(k)];
    const C zm = Z[FL::out_pos((Px - k) % Px)];
    C v;
    if (!im) { v.x = zk.x + zm.x; v.y = zk.y - zm.y; }
    else { v.x = zk.y + zm.y; v.y = zm.x - zk.x; }
    prow<C>(out, fl, row)[k] = v * sc;
  }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
template <typename C> struct ZTile;
// TX x TY lines per CTA: TX runs of the streamwise index (64 B) on the row
// side, TY runs of the wall-normal index on the pencil side; small enough
// for three CTAs per SM.
template <> struct ZTile<double2> { enum { TX = 4, TY = 2 }; };
template <> struct ZTile<float2> { enum { TX = 8, TY = 2 }; };

namespace {
// cuTensorMapEncodeTiled from the driver, looked up once (no -lcuda)
inline PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)p;
  }();
  return fn;
}
// 4-D map (y, kx, kz, field) over 8-byte pencil elements, box 2 x 1 x Nz x 1
inline bool pencil_tmap(const PencilArr& in, int nf, const DnsGeom& g, size_t esz, CUtensorMap* m) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
  if (!enc || esz != 8 || !aligned16(in.base) || (in.ps * esz) % 16 || (in.fs * esz) % 16 || g.Nz > 256)
    return false;
  const cuuint64_t dims[4] = {(cuuint64_t)g.Py, (cuuint64_t)g.Kx, (cuuint64_t)g.Nz, (cuuint64_t)nf};
  const cuuint64_t strides[3] = {(cuuint64_t)(in.ps * esz), (cuuint64_t)((long long)g.Kx * in.ps * esz),
                                 (cuuint64_t)(in.fs * esz)};
  const cuuint32_t box[4] = {2, 1, (cuuint32_t)g.Nz, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, in.base, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// 4-D map (kx, zp, y, field) over 8-byte row elements, box 2 x rows x 1 x 1
inline bool row_tmap(const RowArr& in, int nf, const DnsGeom& g, size_t esz, int rows, CUtensorMap* m) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
  if (!enc || esz != 8 || !aligned16(in.base) || (in.rs * esz) % 16 || (in.fs * esz) % 16 || g.Pz % rows || rows > 256)
    return false;
  const cuuint64_t dims[4] = {(cuuint64_t)g.Kx, (cuuint64_t)g.Pz, (cuuint64_t)g.Py, (cuuint64_t)nf};
  const cuuint64_t strides[3] = {(cuuint64_t)(in.rs * esz), (cuuint64_t)((long long)g.Pz * in.rs * esz),
                                 (cuuint64_t)(in.fs * esz)};
  const cuuint32_t box[4] = {2, (cuuint32_t)rows, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, in.base, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

template <typename C>
cudaError_t launch_zb(PencilArr in, RowArr out, int nf, DnsGeom g, FftTab<C> tab, cudaStream_t st,
                      int* status, int variant, bool probe) {
  const int TX = ZTile<C>::TX, TY = ZTile<C>::TY;
  const bool any = variant == VAR_AUTO;
  if constexpr (sizeof(C) == 8) {
    if (any || variant == DNS_Z_TENSOR_COPY) {
      const cudaError_t e = with_len_z(g.Pz, [&](auto LL) -> cudaError_t {
        constexpr int L = decltype(LL)::value;
        typedef ZStage<C, L> Z;
        if constexpr (Z::ok && Z::fits(L / 3 * 2)) {
          CUtensorMap tm;
          if (status && g.Nz == L / 3 * 2 && tab.zt && pencil_tmap(in, nf, g, sizeof(C), &tm)) {
            if (probe) return cudaSuccess;
            const size_t sm = (size_t)8 * Z::WS * sizeof(C);
            cudaFuncSetAttribute(k_zbt<C, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            dim3 grid((g.Kx - 1 + 7) / 8, (g.Py + 1) / 2, nf);
            k_zbt<C, L><<<grid, 256, sm, st>>>(tm, out, g, tab.zt, status);
            return cudaGetLastError();
          }
        }
        return cudaErrorNotSupported;
      });
      if (e != cudaErrorNotSupported) return e;
    }
  }
  if (any || variant == DNS_Z_WARP) {
    const cudaError_t e = launch_zb2<C>(in, out, nf, g, tab, st, probe);
    if (e != cudaErrorNotSupported) return e;
  }
  if (!any && variant != DNS_Z_BLOCK) return cudaErrorNotSupported;
  if (probe) return cudaSuccess;
  return with_len_xz(g.Pz, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    const size_t sm = (size_t)TX * TY * FLine<C, L>::stride(g.Pz) * sizeof(C);
    cudaFuncSetAttribute(k_zb<C, TX, TY, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    dim3 grid((g.Kx + TX - 1) / TX, (g.Py + TY - 1) / TY, nf);
    k_zb<C, TX, TY, L><<<grid, 256, sm, st>>>(in, out, g, tab);
    return cudaGetLastError();
  });
}
template <typename C>
cudaError_t launch_zf(RowArr in, PencilArr out, int nf, DnsGeom g, FftTab<C> tab, cudaStream_t st,
                      int* status, int variant, bool probe) {
  const int TX = ZTile<C>::TX, TY = ZTile<C>::TY;
  const bool any = variant == VAR_AUTO;
  if constexpr (sizeof(C) == 8) {
    if (any || variant == DNS_Z_TENSOR_COPY) {
      const cudaError_t e = with_len_z(g.Pz, [&](auto LL) -> cudaError_t {
        constexpr int L = decltype(LL)::value;
        typedef ZStage<C, L> Z;
        if constexpr (Z::ok && Z::fits(L) && Z::copies_ok) {
          CUtensorMap tm;
          if (status && g.Nz == L / 3 * 2 && tab.zt && row_tmap(in, nf, g, sizeof(C), Z::ROWS, &tm)) {
            if (probe) return cudaSuccess;
            const size_t sm = (size_t)8 * Z::WS * sizeof(C);
            cudaFuncSetAttribute(k_zft<C, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            dim3 grid((g.Kx + 3) / 4, (g.Py + 3) / 4, nf);
            k_zft<C, L><<<grid, 256, sm, st>>>(tm, out, g, tab.zt, status);
            return cudaGetLastError();
          }
        }
        return cudaErrorNotSupported;
      });
      if (e != cudaErrorNotSupported) return e;
    }
  }
  if (any || variant == DNS_Z_WARP) {
    const cudaError_t e = launch_zf2<C>(in, out, nf, g, tab, st, probe);
    if (e != cudaErrorNotSupported) return e;
  }
  if (!any && variant != DNS_Z_BLOCK) return cudaErrorNotSupported;
  if (probe) return cudaSuccess;
  return with_len_xz(g.Pz, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    const size_t sm = (size_t)TX * TY * FLine<C, L>::stride(g.Pz) * sizeof(C);
    cudaFuncSetAttribute(k_zf<C, TX, TY, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    dim3 grid((g.Kx + TX - 1) / TX, (g.Py + TY - 1) / TY, nf);
    k_zf<C, TX, TY, L><<<grid, 256, sm, st>>>(in, out, g, tab);
    return cudaGetLastError();
  });
}
// CTAs per SM that k_x2 is compiled for, measured at 384 (FP32 / FP64, us):
// five 298 / 644, four 312 / 659; FP32 at 216: seven 33.1, five 34.7; at 96 ten
// 95, seven 99.  Radix 18 in the middle needs the registers of four.
template <typename C, int L> constexpr int x2_ctas() {
  typedef XPlan<L, FftMaxRadix<C>::v> P;
  return P::NW > 3 ? (L > 576 ? 1 : 2) : (P::RF > 16 ? 4 : sizeof(C) == 16 || L >= 256 ? 5 : L > 96 ? 7 : 10);
}
template <typename C, int L, int SC>
cudaError_t launch_x2(RowArr in, RowArr out, DnsGeom g, FftTab<C> tab, const double* Uy, double Ro, int* status,
                      cudaStream_t st, const double* runs) {
  typedef XPlan<L, FftMaxRadix<C>::v> P;
  constexpr int NR = SC * P::NR;
  auto k = k_x2<C, L, SC, (x2_ctas<C, L>() / SC > 0 ? x2_ctas<C, L>() / SC : 1)>;
  const size_t sm = (size_t)3 * NR * xline<C>(L) * sizeof(C);
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  const long long nrows = (long long)g.Py * g.Pz * g.nrun;
  k<<<(unsigned)((nrows + NR - 1) / NR), 32 * SC * P::NW, sm, st>>>(
      in, out, g, tab.xt, Uy, Ro, runs, status);
  return cudaGetLastError();
}
#define DNS_XCASE(n) case n: return f(std::integral_constant<int, n>());
template <typename F> cudaError_t with_len_x(int L, F&& f) {
  switch (L) { XPLAN_LENGTHS(DNS_XCASE) }
  return cudaErrorNotSupported;
}
template <typename C>
cudaError_t launch_x_fused(RowArr in, RowArr out, DnsGeom g, FftTab<C> tab, const double* Uy,
                           double Ro, int* status, cudaStream_t st, int variant, bool probe,
                           const double* runs) {
  const bool any = variant == VAR_AUTO;
  const long long nrows = (long long)g.Py * g.Pz * g.nrun;
  // the fused form stages half spectra of roundup(Nx/2, 8) bins by bulk
  // copies; the rows of a pair share a plane where Pz is even
  const int sr = (g.Nx / 2 + 7) / 8 * 8;
  const bool ok = g.Pz % 2 == 0 && g.Nx / 2 == g.Px / 3 && in.rs >= sr && (in.rs * sizeof(C)) % 16 == 0 &&
                  (in.fs * sizeof(C)) % 16 == 0 && aligned16(in.base) && status && nrows < (1LL << 31) &&
                  tab.xt;
  if (ok && (any || variant == DNS_X_WARP3 || variant == DNS_X_WARP6)) {
    const cudaError_t e = with_len_x(g.Px, [&](auto LL) -> cudaError_t {
      constexpr int L = decltype(LL)::value;
      if (variant == DNS_X_WARP6) {
        // two row groups per CTA, for the lengths of the named grids
        if constexpr (L == 48 || L == 96 || L == 144 || L == 192 || L == 384) {
          return probe ? cudaSuccess : launch_x2<C, L, 2>(in, out, g, tab, Uy, Ro, status, st, runs);
        }
        return cudaErrorNotSupported;
      }
      return probe ? cudaSuccess : launch_x2<C, L, 1>(in, out, g, tab, Uy, Ro, status, st, runs);
    });
    if (e != cudaErrorNotSupported) return e;
  }
  if (!any && variant != DNS_X_BLOCK) return cudaErrorNotSupported;
  if (probe) return cudaSuccess;
  return with_len_xz(g.Px, [&](auto LL) -> cudaError_t {
    constexpr int L = decltype(LL)::value;
    const size_t sm = (size_t)(L > 0 ? 6 : 9) * FLine<C, L>::stride(g.Px) * sizeof(C);
    cudaFuncSetAttribute(k_x_fused<C, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    const long long pairs = ((long long)g.Py * g.Pz + 1) / 2 * g.nrun;
    k_x_fused<C, L><<<(unsigned)pairs, 256, sm, st>>>(in, out, g, tab, Uy, Ro, runs);
    return cudaGetLastError();
  });
}
