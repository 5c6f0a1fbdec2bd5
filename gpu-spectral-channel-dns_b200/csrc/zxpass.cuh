// Launchers of the spanwise / streamwise pass kernels (zxstep.cuh; the drop-ins zxpass.cu).
#pragma once
#include "kernels.cuh"

template <typename C>
cudaError_t launch_zb(PencilArr in, RowArr out, int nf, DnsGeom g, FftTab<C> tab, cudaStream_t st,
                      int* status = nullptr, int variant = VAR_AUTO, bool probe = false);
template <typename C>
cudaError_t launch_zf(RowArr in, PencilArr out, int nf, DnsGeom g, FftTab<C> tab, cudaStream_t st,
                      int* status = nullptr, int variant = VAR_AUTO, bool probe = false);
template <typename C>
cudaError_t launch_x_fused(RowArr in, RowArr out, DnsGeom g, FftTab<C> tab, const double* Uy,
                           double Ro, int* status, cudaStream_t st, int variant = VAR_AUTO,
                           bool probe = false, const double* runs = nullptr);
// FP64 pieces of the reference-layout transforms, nf <= 6 fields a launch:
// rows (field by field, stride fs) to fields of points and back (x scale; the
// Kx bins that the spanwise pass reads), and the spanwise passes
cudaError_t launch_x_c2r(RowArr in, FieldList out, int nf, long long rps, long long nrows, DnsGeom g,
                         FftTab<double2> tab, cudaStream_t st);
cudaError_t launch_x_r2c(FieldList in, int nf, long long rps, RowArr out, long long nrows, DnsGeom g,
                         FftTab<double2> tab, double scale, cudaStream_t st);
cudaError_t launch_zb_fields(PencilList in, RowArr out, int nf, DnsGeom g, FftTab<double2> tab, cudaStream_t st,
                             int variant = VAR_AUTO);
cudaError_t launch_zf_fields(RowArr in, PencilList out, int nf, DnsGeom g, FftTab<double2> tab, cudaStream_t st,
                             int variant = VAR_AUTO);
cudaError_t launch_lamb_rows(const double* const in6[6], double* const out3[3], long long rps,
                             long long nrows, DnsGeom g, const double* Uy, double Ro,
                             cudaStream_t st);
