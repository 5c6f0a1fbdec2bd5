// The FP64 spanwise and streamwise passes of the time step.
#include "zxstep.cuh"

template cudaError_t launch_zb<double2>(PencilArr, RowArr, int, DnsGeom, FftTab<double2>, cudaStream_t, int*, int, bool);
template cudaError_t launch_zf<double2>(RowArr, PencilArr, int, DnsGeom, FftTab<double2>, cudaStream_t, int*, int, bool);
template cudaError_t launch_x_fused<double2>(RowArr, RowArr, DnsGeom, FftTab<double2>, const double*,
                                         double, int*, cudaStream_t, int, bool, const double*);
