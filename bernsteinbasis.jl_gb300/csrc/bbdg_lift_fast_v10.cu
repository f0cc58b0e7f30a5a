// FP32 lift kernels for N = 10, 11.
#include "bbdg_lift_fast_impl.cuh"

template int bblift::launch_lift4<10>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
template int bblift::launch_lift4<11>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
