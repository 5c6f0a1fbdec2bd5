// The FP32 (mixed form) spanwise and streamwise passes of the time step.
#include "zxstep.cuh"

template cudaError_t launch_zb<float2>(PencilArr, RowArr, int, DnsGeom, FftTab<float2>, cudaStream_t, int*, int, bool);
template cudaError_t launch_zf<float2>(RowArr, PencilArr, int, DnsGeom, FftTab<float2>, cudaStream_t, int*, int, bool);
template cudaError_t launch_x_fused<float2>(RowArr, RowArr, DnsGeom, FftTab<float2>, const double*,
                                         double, int*, cudaStream_t, int, bool, const double*);
