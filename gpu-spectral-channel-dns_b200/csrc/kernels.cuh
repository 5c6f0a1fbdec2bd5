// Kernel parameter blocks and launch helpers shared by the pass kernels.
//
// Layouts (element = complex of the pass precision unless stated):
//   pencil arrays  [field][pencil][n]     pencil p = kz*Kx + kx, wall-normal
//                                         index n contiguous (pitch ps); this
//                                         is the reference's ZXY layout
//                                         (include/data.h:265-284) when ps is
//                                         tPitch/16 and the field stride is 0
//   row arrays     [field][y][zp][kx]     streamwise index contiguous (row
//                                         pitch rs, Pz rows per wall-normal
//                                         plane); the reference's XYZ complex
//                                         layout before its 2D C2R
//   state arrays   [pencil][n] FP64 complex, n < Ny, pitch Ny
#pragma once
#include "../../include/dns_b200.h"
#include "dns_common.cuh"
#include "fft.cuh"

template <typename C> struct FftTab {
  FftPlan plan;
  const C* tw;          // W_L^j, j < L
  const short* drev;    // digit-reversed position of natural index n
  const C* dt;          // twiddles of the pruned DCT (ydct.cuh), null for lengths without one
  const C* xt;          // twiddles of the fused streamwise form (xpass.cuh), null for lengths without one
  const C* zt;          // twiddles of the two-pass spanwise form (zpass.cuh), null for lengths without one
};

// Pass launchers take a variant (the DNS_Y3_*, DNS_Y1_*, DNS_Z_* values of
// the public header) or VAR_AUTO, the first form the arguments allow in the
// order tensor copies, warp FFTs, block FFT.  With a variant they launch
// exactly that form or return cudaErrorNotSupported; with probe = true they
// only report which of the two it would be.
#define VAR_AUTO (-1)

struct PencilArr {      // generic pencil-major array
  void* base;
  long long ps;         // pencil pitch (elements)
  long long fs;         // field stride (elements)
};

struct FieldList {      // up to six fields, anywhere
  void* p[6];
};
struct PencilList {     // pencil-major fields, anywhere
  FieldList f;
  long long ps;         // pencil pitch (elements)
};
// field f of either form
template <typename C> DNS_HD C* field_base(const PencilArr& a, int f) { return (C*)a.base + (long long)f * a.fs; }
template <typename C> DNS_HD C* field_base(const PencilList& a, int f) { return (C*)a.f.p[f]; }

struct RowArr {         // generic row-major [field][y][zp][kx] array
  void* base;
  long long rs;         // row pitch (elements)
  long long fs;         // field stride (elements)
};

// default bound of a device wait, in SM clock cycles (~1 s at 2 GHz)
#define DNS_WAIT_LIMIT (1LL << 31)

struct PhysParams {
  double aphi, beta;    // box: alpha_k = kx/aphi, beta_k = kz/beta
  double Re, Ro, dt;
  double U0, U1, U2;    // base flow U(y) = U0 + U1 y + U2 y^2
  long long wait_limit = DNS_WAIT_LIMIT;  // staging waits of the wall-normal warp passes
  const double* runs = nullptr;  // a batch's per-member (Re, Ro, dt), 3 each; null: one run
};
// a batch member's parameters (the context's own for one run)
DNS_HD double run_Re(const PhysParams& ph, int r) { return ph.runs ? ph.runs[3 * r] : ph.Re; }
DNS_HD double run_Ro(const PhysParams& ph, int r) { return ph.runs ? ph.runs[3 * r + 1] : ph.Ro; }
DNS_HD double run_dt(const PhysParams& ph, int r) { return ph.runs ? ph.runs[3 * r + 2] : ph.dt; }

// 16-byte alignment of a device pointer (bulk-copy sources)
inline bool aligned16(const void* p) { return ((unsigned long long)p & 15ull) == 0; }
// whether a kernel on device dev can take p for complex loads, a the runtime's
// attributes of p: dev's own or managed memory.  Another device's memory is for
// copies only (without peer access a kernel faults on it), as is the host's.
inline bool kernel_memory(const void* p, const cudaPointerAttributes& a, int dev) {
  return aligned16(p) && ((a.type == cudaMemoryTypeDevice && a.device == dev) || a.type == cudaMemoryTypeManaged);
}
// n rows of w bytes, pitch bytes apart
struct PitchedBytes {
  const void* p;
  long long n, w, pitch;
  const char* end() const { return (const char*)p + (n - 1) * pitch + w; }
};
// whether two of them share a byte (those of one pitch may interleave their rows)
inline bool rows_overlap(const PitchedBytes& a, const PitchedBytes& b) {
  if ((const char*)a.p >= b.end() || (const char*)b.p >= a.end()) return false;
  if (a.pitch != b.pitch) return true;
  const long long d = ((const char*)b.p - (const char*)a.p) % a.pitch, r = d < 0 ? d + a.pitch : d;
  return r < a.w || a.pitch - r < b.w;
}
// whether the fields of one transform call can share launches: no field's output
// lies in another's input or output.  Fields that do go one by one, in order.
inline bool fields_apart(bool forward, int nf, const PitchedBytes* phys, const PitchedBytes* spec) {
  for (int i = 0; i < nf; ++i)
    for (int j = 0; j < nf; ++j) {
      if (i == j) continue;
      // (the pencils are overwritten in both directions)
      if (rows_overlap(spec[i], phys[j]) || (i < j && rows_overlap(spec[i], spec[j]))) return false;
      if (!forward && i < j && rows_overlap(phys[i], phys[j])) return false;
    }
  return true;
}

#define DNS_CHECK_LAUNCH() do { cudaError_t e__ = cudaGetLastError(); if (e__ != cudaSuccess) return e__; } while (0)
