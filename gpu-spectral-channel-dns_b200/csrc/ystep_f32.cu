// The mixed (FP32 transforms) wall-normal passes of the time step.
#include "ystep.cuh"

template cudaError_t launch_y3<float2>(const double2*, const double2*, PencilArr, DnsGeom, PhysParams, FftTab<float2>, int*, cudaStream_t, int, bool);
template cudaError_t launch_y1<float2>(PencilArr, const double2*, const double2*, double2*, double2*, double2*, double2*, RhsDims, RhsTabs, DnsGeom, PhysParams, FftTab<float2>, int, int*, cudaStream_t, int, bool);
