// FP32 lift kernels for N = 12, 13, 14, 15.
#include "bbdg_lift_fast_impl.cuh"

template int bblift::launch_lift4<12>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
template int bblift::launch_lift4<13>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
template int bblift::launch_lift4<14>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
template int bblift::launch_lift4<15>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
