// Per-step wall-normal solves (the y2 kernel): v solve, tilting term,
// omega_y solve, for every Fourier mode, on the banded integrated systems of
// wallsolve.h.  Replaces the reference's explicit-inverse products
// (source/solver.cpp:107-123, matrix_op.cpp:68-78) and the tilting term of
// _get_linear_omega_y (source/linear.cpp:147-151).
//
// One CTA = one warp = a group of 16 operator slots; lane 2q + b handles
// pencil b (kz' or Nz - kz') of slot q, both pencils sharing the slot's
// factors.  The factors of a group are stored as one contiguous stream in
// the order the solve reads them (v forward rows, v backward rows, omega
// forward rows, omega backward rows; each row holds its entries for the 16
// slots side by side), and are streamed through a shared-memory ring with
// cp.async.bulk and mbarriers.  Each lane keeps its intermediate solution
// and tilting term in one column of a global scratch of the group (rows
// interleaved over the lanes, L2-resident, one ring chunk of rows in
// registers ahead of the recurrence), so that a CTA needs only the ring and two small tables in
// shared memory and several CTAs share an SM.
//
// Inputs from the y1 kernel: g_v, g_o (rows K.. of the integrated
// collocation right-hand sides, the v^n part of the tilting term included).
// Outputs: V, O (Chebyshev coefficients of v^{n+1}, omega_y^{n+1}); the
// solve-only entry adds its wall polynomials (pbc) to the lowest ones.
#include "kernels.cuh"
#include "mbar.cuh"
#include "wallsolve_dev.cuh"

#define WALL_WAIT_LIMIT (1LL << 31)

namespace {

constexpr int WALL_HDR = 128;        // mbarriers

// Variants (the solve's tunable block shape): ring stages, bytes per stage
// and whether the tilting table sits in shared memory (else read through L1).
// The factor stream is read with the L2 evict-first policy (the scratch vectors
// then stay in L2).  More rows per stage hide the scratch loads of a warp, a
// smaller ring leaves room for more CTAs per SM.
struct WallVar {
  int nst, stg;
  bool qsm;
};
constexpr WallVar kWallVar[DNS_WALL_VARIANTS] = {{2, 24576, true}, {2, 18432, true}, {2, 12288, false}, {2, 16384, true}};

__host__ __device__ constexpr int rows_per_chunk(int stg, int entries, int cap) {
  return (stg / (entries * 256)) < cap ? (stg / (entries * 256)) : cap;
}

// acc - a b: four fused operations (a product and a sum apart are six)
__device__ __forceinline__ double2 cfms(double2 a, double2 b, double2 acc) {
  return make_double2(fma(a.y, b.y, fma(-a.x, b.x, acc.x)), fma(-a.y, b.x, fma(-a.x, b.y, acc.y)));
}
__device__ __forceinline__ double2 rfma(double a, double2 b, double2 acc) {
  return make_double2(fma(a, b.x, acc.x), fma(a, b.y, acc.y));
}

template <int KLV, int KUV, int KLO, int KUO, int STG>
struct WallCfg {
  static constexpr int E0 = KLV, E1 = 1 + KUV + 2, E2 = KLO, E3 = 1 + KUO;
  // rows per ring chunk; the solve keeps a chunk of vector rows in registers
  static constexpr int R0 = rows_per_chunk(STG, E0, WALL_ROWS), R1 = rows_per_chunk(STG, E1, WALL_ROWS);
  static constexpr int R2 = rows_per_chunk(STG, E2, WALL_ROWS), R3 = rows_per_chunk(STG, E3, WALL_ROWS);
  static_assert(R0 > 0 && R1 > 1 && R2 > 0 && R3 > 0, "stage too small for a row");
};

}  // namespace

template <int KLV, int KUV, int KLO, int KUO, int WALL_NST, int WALL_STG, bool QSM>
__global__ void __launch_bounds__(32) k_wall_solve(const double2* __restrict__ fac, double2* V,
                                                   double2* O, const double2* __restrict__ gv,
                                                   const double2* __restrict__ go,
                                                   const double* __restrict__ Qg, double2* Sw,
                                                   const double2* __restrict__ pbc, WallDims wd, DnsGeom g, PhysParams ph, int* status) {
  typedef WallCfg<KLV, KUV, KLO, KUO, WALL_STG> CF;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* full = (uint64_t*)smem_raw;
  double2* ring = (double2*)(smem_raw + WALL_HDR);
  double* Qsm = (double*)(smem_raw + WALL_HDR + WALL_NST * WALL_STG);
  const double* Qs = (QSM ? Qsm : Qg) + 7 * WALL_QLOW;  // tilting table: shared memory or through L1
  // recombination weights of the clamped basis, row by row
  double* rc2 = Qsm + (QSM ? wd.qbytes / 8 : 0);
  double* rc4 = rc2 + wd.nv + WALL_ROWS;

  const int lane = threadIdx.x;
  const int q = lane >> 1, b = lane & 1;
  // member of a batch (its groups are consecutive CTAs)
  const long long gpr = wd.groups_per_run > 0 ? wd.groups_per_run : (long long)gridDim.x;
  const int run = (int)(blockIdx.x / gpr);
  const long long slot = ((long long)blockIdx.x - run * gpr) * 16 + q;
  const bool valid = slot < wd.nslots;
  const int kx = valid ? (int)(slot % g.Kx) : 0;
  const int kzs = valid ? wd.kzs0 + (int)(slot / g.Kx) : 0;
  const int npen = (kzs == 0 || kzs == g.Nz / 2) ? 1 : 2;
  const bool active = valid && b < npen;
  const int kz = (b == 0) ? kzs : g.Nz - kzs;
  const long long pen = (long long)run * g.Hrun +
                        ((b == 0) ? wd.rowa + (long long)(kz - wd.kza) * g.Kx + kx
                                  : wd.rowb + (long long)(kz - wd.kzb) * g.Kx + kx);
  const bool zero = valid && kzs == 0 && kx == 0;
  double ia, ib;
  wavenumbers(kx, kz, g.Nz, ph.aphi, ph.beta, ia, ib);
  const double kap = (zero || !wd.tilt) ? 0.0 : -0.5 * ib * run_dt(ph, run);  // tilting weight of this pencil
  const int N = g.Ny - 1;
  // this lane's vector (right-hand side, intermediate solution, tilting
  // term) in the group's scratch, rows interleaved over the 32 lanes: a
  // row of the warp is one contiguous 512-byte access
  double2* S = Sw + (long long)blockIdx.x * 32 * wd.nv + lane;
  const double2 z2 = make_double2(0.0, 0.0);
  const double2* gfac = fac + (long long)blockIdx.x * wd.group_complex;
  const int nch0 = (wd.nv + CF::R0 - 1) / CF::R0, nch1 = (wd.nv + CF::R1 - 1) / CF::R1;
  const int nch2 = (wd.no + CF::R2 - 1) / CF::R2, nch3 = (wd.no + CF::R3 - 1) / CF::R3;
  const bool dov = wd.sys & 1, doo = wd.sys & 2;
  const int total = (dov ? nch0 + nch1 : 0) + (doo ? nch2 + nch3 : 0);

  const uint64_t pol = l2_evict_first();
  // the group's stream is contiguous: lane 0 walks it phase by phase, ic the
  // next chunk, irow rows of its phase issued.  Rows ascend in phases 0 and 2,
  // whose last chunk may be short; they descend in phases 1 and 3, whose first
  // one may be, its rows at the end of the stage.
  const int n1 = (wd.nv - 1) % CF::R1 + 1, n3 = (wd.no - 1) % CF::R3 + 1;
  int ic = 0, iph = dov ? 0 : 2, irow = 0;
  const double2* isrc = gfac + (dov ? 0 : 16LL * wd.nv * (CF::E0 + CF::E1));
  auto issue = [&]() {
    const int rows = iph < 2 ? wd.nv : wd.no;
    const int R = iph == 0 ? CF::R0 : iph == 1 ? CF::R1 : iph == 2 ? CF::R2 : CF::R3;
    const int E = iph == 0 ? CF::E0 : iph == 1 ? CF::E1 : iph == 2 ? CF::E2 : CF::E3;
    int n = min(R, rows - irow);
    uint64_t* bar = &full[ic % WALL_NST];
    double2* dst = ring + (size_t)(ic % WALL_NST) * (WALL_STG / 16);
    if ((iph & 1) && irow == 0) {
      n = iph == 1 ? n1 : n3;
      dst += (R - n) * E * 16;
    }
    const uint32_t bytes = (uint32_t)(n * E * 256);
    mbar_expect_tx(bar, bytes);
    bulk_g2s_hint(dst, isrc, bytes, bar, pol);
    isrc += n * E * 16;
    irow += n;
    if (irow == rows) { irow = 0; ++iph; }
    ++ic;
  };
  // on a timed-out wait: report, let the copies in flight land, leave
  auto abort_at = [&](int c) {
    if (lane == 0) {
      atomicOr(status, 1);
      for (int cc = c; cc < min(c + WALL_NST, total); ++cc)
        mbar_wait_bounded(&full[cc % WALL_NST], (uint32_t)((cc / WALL_NST) & 1), WALL_WAIT_LIMIT, nullptr);
    }
  };
  auto wait_chunk = [&](int c) {
    const bool ok = mbar_wait_bounded(&full[c % WALL_NST], (uint32_t)((c / WALL_NST) & 1),
                                      WALL_WAIT_LIMIT, status);
    return __all_sync(0xffffffffu, ok);
  };
  auto release = [&]() {
    __syncwarp();
    if (lane == 0 && ic < total) {
      fence_proxy_async();
      issue();
    }
  };
  auto chunk_at = [&](int c) { return ring + (size_t)(c % WALL_NST) * (WALL_STG / 16) + q; };
  // zeros before the rows of a descending phase's short first chunk: those rows,
  // above the last, then come out as zeros
  auto zero_rows = [&](int c, int n) {
    double2* z = ring + (size_t)(c % WALL_NST) * (WALL_STG / 16);
    for (int k = lane; k < n * 16; k += 32) z[k] = z2;
    fence_proxy_async();
    __syncwarp();
  };
  const double2* gvp = gv + pen * wd.gp;
  const double2* gop = go + pen * wd.gp;
  const int nv = wd.nv, no = wd.no;

  // ---- start: barriers, ring prefetch, tables ----------------------------
  if (lane == 0) {
    for (int s = 0; s < WALL_NST; ++s) mbar_init(&full[s], 1);
    fence_mbar_init();
  }
  __syncwarp();
  if (QSM)
    for (int k = lane; k < WALL_QROWS(no) * 7; k += 32) Qsm[k] = Qg[k];
  // recombination weights of row i: V_{i+4} = x_{i+4} - 2k/(k+1) x_{i+2} +
  // (k-3)/(k-1) x_i, k = i + 4, unknowns from N - 3 on are not part of it
  for (int i = lane; i < nv + WALL_ROWS; i += 32) {
    const int k = i + 4;
    rc2[i] = i + 2 < N - 3 ? 2.0 * k / (k + 1) : 0.0;
    rc4[i] = i < N - 3 ? (double)(k - 3) / (double)(k - 1) : 0.0;
  }
  if (lane == 0)
    for (int c = 0; c < min(WALL_NST, total); ++c) issue();
  __syncwarp();
  // the group of the mean modes (two systems of the omega kind)
  const bool mean = __any_sync(0xffffffffu, zero);

  // Rows go in chunks of the ring; a row's vector element is loaded one chunk
  // ahead into the register it is consumed from.  Every chunk runs the same
  // code without conditions between its rows, so that the windows of earlier
  // rows are renamed registers and not moves: rows beyond a phase's last are
  // computed and not stored (ascending) or come first as zeros (descending).
  // One body per phase: a warp is alone on its scheduler, and a grid of few
  // groups spends a third of its time fetching instructions.
  int c = 0;
  // ---- v: forward substitution (unit lower band) -------------------------
  if (dov) {
    constexpr int R = CF::R0;
    double2 yw[KLV], cur[R];
#pragma unroll
    for (int e = 0; e < KLV; ++e) yw[e] = z2;
#pragma unroll
    for (int rr = 0; rr < R; ++rr) cur[rr] = (active && rr < nv) ? __ldg(gvp + rr) : z2;
    auto chunk = [&](const double2* ch, int r0) {
      const double2* nx = gvp + r0 + R;
      double2* Sr = S + 32 * r0;
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        const double2* Lr = ch + rr * CF::E0 * 16;
        // the older entries in independent partial sums; the newest
        // (y_{i-1}) last, so only it is on the row-to-row critical path
        double2 a0 = cur[rr], a1 = z2;
        cur[rr] = (active && r0 + R + rr < nv) ? __ldg(nx + rr) : z2;
#pragma unroll
        for (int e = 0; e < KLV - 1; ++e) {
          if (e & 1) a1 = cfms(Lr[e * 16], yw[e], a1);
          else a0 = cfms(Lr[e * 16], yw[e], a0);
        }
        const double2 acc = cfms(Lr[(KLV - 1) * 16], yw[KLV - 1], a0 + a1);
        if (r0 + rr < nv) Sr[32 * rr] = acc;
#pragma unroll
        for (int e = 0; e < KLV - 1; ++e) yw[e] = yw[e + 1];
        yw[KLV - 1] = acc;
      }
    };
    for (int r0 = 0; r0 < nv; r0 += R, ++c) {
      if (!wait_chunk(c)) { abort_at(c); return; }
      chunk(chunk_at(c), r0);
      release();
    }
  }
  // ---- v: back substitution, recombination, tilting term -----------------
  // rows descend.  The tilting term of row k+1 is written over rows already
  // consumed (k + 1 > i).
  if (dov) {
    constexpr int R = CF::R1;
    double2 xw[KUV], cur[R];
#pragma unroll
    for (int e = 0; e < KUV; ++e) xw[e] = z2;
    double2 xd0 = z2, xd1 = z2;
    double2 P[7];  // P[j]: partial tilting sum of row k+1-j, k = next coefficient emitted
#pragma unroll
    for (int j = 0; j < 7; ++j) P[j] = z2;
    // base-flow degree (KLV = deg U + 4): U' = U1 (degree 1) makes the
    // tilting operator B^2 U1, three diagonals; U' = 0 (degree 0) none
    constexpr int DEG = KLV - 4;
    // coefficient k into the tilting sums, row k + 1 of the term out; the
    // table has zero rows around it (FIRST: rows below 0 beyond those)
    auto tilt = [&](int k, double2 a, bool first) {
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        if (DEG == 0 || (DEG == 1 && (j & 1) == 0)) continue;
        const int r = k + 1 - j;
        if (!first || r >= 0) P[j] = rfma(QSM ? Qs[7 * r + j] : __ldg(Qs + 7 * r + j), a, P[j]);
      }
      if (k + 1 < no) S[32 * (k + 1)] = make_double2(-P[0].y * kap, P[0].x * kap);
#pragma unroll
      for (int j = 0; j < 6; ++j) P[j] = P[j + 1];
      P[6] = z2;
    };
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      const int i = nch1 * R - 1 - rr;
      cur[rr] = i < nv ? S[32 * i] : z2;
    }
    double2* Vp = V + pen * wd.xp + (zero ? 2 : 4);  // row i emits coefficient i + 4, of the mean modes i + 2
    const int top = zero ? N - 2 : N - 4;         // the last row that emits one
    auto chunk = [&](const double2* ch, int i0) {
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        const int i = i0 - rr;
        const double2* Ur = ch + rr * CF::E1 * 16;
        double2 a0 = cur[rr];
        cur[rr] = i >= R ? S[32 * (i - R)] : z2;
        // independent partial sums; x_{i+1} enters last
        double2 a1 = z2, a2 = z2;
        a1 = cfms(Ur[(KUV + 1) * 16], xd0, a1);
        a2 = cfms(Ur[(KUV + 2) * 16], xd1, a2);
#pragma unroll
        for (int e = KUV; e >= 2; --e) {
          if (e % 3 == 0) a1 = cfms(Ur[e * 16], xw[e - 1], a1);
          else if (e % 3 == 1) a2 = cfms(Ur[e * 16], xw[e - 1], a2);
          else a0 = cfms(Ur[e * 16], xw[e - 1], a0);
        }
        const double2 acc = cfms(Ur[16], xw[0], a0 + (a1 + a2));
        const double2 x = cmul(Ur[0], acc);
        if (i >= nv - 2) {  // the two unknowns with dense columns
          if (i == nv - 1) xd1 = x;
          if (i == nv - 2) xd0 = x;
        }
#pragma unroll
        for (int e = KUV - 1; e >= 1; --e) xw[e] = xw[e - 1];
        xw[0] = x;
        double w2 = rc2[i], w4 = rc4[i], w0 = i + 4 < N - 3 ? 1.0 : 0.0;
        if (mean && zero) {
          w2 = i + 2 < N - 1 ? 1.0 : 0.0;
          w4 = i < N - 1 ? 1.0 : 0.0;
          w0 = 0.0;
        }
        const double2 a = rfma(w4, x, rfma(-w2, xw[2], xw[4] * w0));
        if (active && i <= top) Vp[i] = a;
        tilt(i + 4, a, false);
      }
    };
    for (int i0 = nch1 * R - 1; i0 >= 0; i0 -= R, ++c) {
      if (!wait_chunk(c)) { abort_at(c); return; }
      if (i0 >= nv) zero_rows(c, (R - n1) * CF::E1);
      chunk(chunk_at(c), i0);
      release();
    }
    double2 a[4];
    a[3] = xw[3] - xw[1] * 1.5;
    a[2] = xw[2] - xw[0] * (4.0 / 3.0);
    a[1] = xw[1];
    a[0] = xw[0];
    if (zero) {
      a[1] = make_double2(-xw[1].x, -xw[1].y);
      a[0] = make_double2(-xw[0].x, -xw[0].y);
    }
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      if (active && !(zero && k > 1)) V[pen * wd.xp + k] = pbc ? a[k] + pbc[pen * 6 + k] : a[k];
      tilt(k, a[k], true);
    }
    S[0] = make_double2(-P[0].y * kap, P[0].x * kap);
  }
  if (!doo) return;
  // ---- omega: forward substitution (adds g_o to the tilting term) --------
  {
    constexpr int R = CF::R2;
    double2 ow[KLO], gc[R], sc[R];
#pragma unroll
    for (int e = 0; e < KLO; ++e) ow[e] = z2;
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      gc[rr] = (active && rr < no) ? __ldg(gop + rr) : z2;
      sc[rr] = dov && rr < no ? S[32 * rr] : z2;
    }
    auto chunk = [&](const double2* ch, int r0) {
      const double2* nx = gop + r0 + R;
      double2* Sr = S + 32 * r0;
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        const double2* Lr = ch + rr * CF::E2 * 16;
        double2 a0 = sc[rr] + gc[rr];
        const bool more = r0 + R + rr < no;
        gc[rr] = (active && more) ? __ldg(nx + rr) : z2;
        sc[rr] = dov && more ? Sr[32 * (R + rr)] : z2;
        double2 a1 = z2;
#pragma unroll
        for (int e = 0; e < KLO - 1; ++e) {
          if (e & 1) a1 = cfms(Lr[e * 16], ow[e], a1);
          else a0 = cfms(Lr[e * 16], ow[e], a0);
        }
        const double2 acc = cfms(Lr[(KLO - 1) * 16], ow[KLO - 1], a0 + a1);
        if (r0 + rr < no) Sr[32 * rr] = acc;
#pragma unroll
        for (int e = 0; e < KLO - 1; ++e) ow[e] = ow[e + 1];
        ow[KLO - 1] = acc;
      }
    };
    for (int r0 = 0; r0 < no; r0 += R, ++c) {
      if (!wait_chunk(c)) { abort_at(c); return; }
      chunk(chunk_at(c), r0);
      release();
    }
  }
  // ---- omega: back substitution and recombination ------------------------
  {
    constexpr int R = CF::R3;
    double2 zw[KUO], cur[R];
#pragma unroll
    for (int e = 0; e < KUO; ++e) zw[e] = z2;
    const int nbo = N - 1;
    double2* Op = O + pen * wd.xp + 2;
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      const int i = nch3 * R - 1 - rr;
      cur[rr] = i < no ? S[32 * i] : z2;
    }
    auto chunk = [&](const double2* ch, int i0) {
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        const int i = i0 - rr;
        const double2* Ur = ch + rr * CF::E3 * 16;
        double2 a0 = cur[rr], a1 = z2;
        cur[rr] = i >= R ? S[32 * (i - R)] : z2;
#pragma unroll
        for (int e = KUO; e >= 2; --e) {
          if (e & 1) a1 = cfms(Ur[e * 16], zw[e - 1], a1);
          else a0 = cfms(Ur[e * 16], zw[e - 1], a0);
        }
        const double2 acc = cfms(Ur[16], zw[0], a0 + a1);
        const double2 x = cmul(Ur[0], acc);
#pragma unroll
        for (int e = KUO - 1; e >= 1; --e) zw[e] = zw[e - 1];
        zw[0] = x;
        if (active && i < nbo) Op[i] = rfma(i + 2 < nbo ? -1.0 : 0.0, zw[2], x);
      }
    };
    for (int i0 = nch3 * R - 1; i0 >= 0; i0 -= R, ++c) {
      if (!wait_chunk(c)) { abort_at(c); return; }
      if (i0 >= no) zero_rows(c, (R - n3) * CF::E3);
      chunk(chunk_at(c), i0);
      release();
    }
    if (active) {
      const double2 a1 = make_double2(-zw[1].x, -zw[1].y), a0 = make_double2(-zw[0].x, -zw[0].y);
      O[pen * wd.xp + 1] = pbc ? a1 + pbc[pen * 6 + 5] : a1;
      O[pen * wd.xp + 0] = pbc ? a0 + pbc[pen * 6 + 4] : a0;
    }
  }
}

size_t wall_smem_bytes(const WallDims& wd, int variant) {
  const WallVar& v = kWallVar[variant];
  return (size_t)WALL_HDR + (size_t)v.nst * v.stg + (v.qsm ? wd.qbytes : 0) + (size_t)2 * (wd.nv + WALL_ROWS) * 8;
}
size_t wall_scratch_complex(const WallDims& wd) { return (size_t)wd.ngroups * 32 * wd.nv; }

// band instances: base-flow degree 0, 1, 2
bool wall_band_of(int delta, int* klv, int* kuv, int* klo, int* kuo) {
  static const int tab[3][4] = {{4, 8, 2, 4}, {5, 9, 3, 6}, {6, 10, 4, 8}};
  if (delta < 0 || delta > 2) return false;
  *klv = tab[delta][0]; *kuv = tab[delta][1]; *klo = tab[delta][2]; *kuo = tab[delta][3];
  return true;
}

template <int A, int B, int C, int D, int VAR>
static cudaError_t launch_inst(const double2* fac, double2* V, double2* O, const double2* gv,
                               const double2* go, const double* Q, double2* Sw, const double2* pbc,
                               const WallDims& wd, const DnsGeom& g, const PhysParams& ph, int* status, cudaStream_t st) {
  constexpr WallVar v = kWallVar[VAR];
  auto k = k_wall_solve<A, B, C, D, v.nst, v.stg, v.qsm>;
  const size_t sm = wall_smem_bytes(wd, VAR);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e) return e;
  k<<<(unsigned)wd.ngroups, 32, sm, st>>>(fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status);
  return cudaGetLastError();
}

template <int A, int B, int C, int D>
static cudaError_t launch_var(int variant, const double2* fac, double2* V, double2* O, const double2* gv,
                              const double2* go, const double* Q, double2* Sw, const double2* pbc,
                              const WallDims& wd, const DnsGeom& g, const PhysParams& ph, int* status, cudaStream_t st) {
  switch (variant) {
    case 0: return launch_inst<A, B, C, D, 0>(fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
    case 1: return launch_inst<A, B, C, D, 1>(fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
    case 2: return launch_inst<A, B, C, D, 2>(fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
    case 3: return launch_inst<A, B, C, D, 3>(fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
  }
  return cudaErrorNotSupported;
}

cudaError_t launch_wall_solve(const double2* fac, double2* V, double2* O, const double2* gv,
                              const double2* go, const double* Q, double2* Sw, const WallDims& wd,
                              const DnsGeom& g, const PhysParams& ph, int* status, cudaStream_t st,
                              int variant, const double2* pbc) {
  if (variant < 0 || variant >= DNS_WALL_VARIANTS) return cudaErrorNotSupported;
  if (wall_smem_bytes(wd, variant) > 227 * 1024) return cudaErrorNotSupported;
  switch (wd.delta) {
    case 0: return launch_var<4, 8, 2, 4>(variant, fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
    case 1: return launch_var<5, 9, 3, 6>(variant, fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
    case 2: return launch_var<6, 10, 4, 8>(variant, fac, V, O, gv, go, Q, Sw, pbc, wd, g, ph, status, st);
  }
  return cudaErrorInvalidValue;
}
