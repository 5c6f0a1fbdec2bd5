// The FP64 wall-normal passes of the time step.
#include "ystep.cuh"

template cudaError_t launch_y3<double2>(const double2*, const double2*, PencilArr, DnsGeom, PhysParams, FftTab<double2>, int*, cudaStream_t, int, bool);
template cudaError_t launch_y1<double2>(PencilArr, const double2*, const double2*, double2*, double2*, double2*, double2*, RhsDims, RhsTabs, DnsGeom, PhysParams, FftTab<double2>, int, int*, cudaStream_t, int, bool);
