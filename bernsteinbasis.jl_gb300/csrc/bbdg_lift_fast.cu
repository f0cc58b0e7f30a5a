// Dispatch of the degree-specialised FP32 lift, and its kernels up to degree 9 (the higher
// ones compile in bbdg_lift_fast_v*.cu).
#include "bbdg_lift_fast_impl.cuh"

extern template int bblift::launch_lift4<10>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
extern template int bblift::launch_lift4<11>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
extern template int bblift::launch_lift4<12>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
extern template int bblift::launch_lift4<13>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
extern template int bblift::launch_lift4<14>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);
extern template int bblift::launch_lift4<15>(bb_ctx*, const DegTables*, int64_t, const void*, void*, cudaStream_t);

// FP32 lift of K columns with the degree-specialised kernels; nfaces 4 (BernsteinLift, N <= 15)
// or 1 (face_lift_multiply!, N <= 12). Returns -1 when no specialised kernel applies (degree
// above those, or a 4-face input or output that is not 16-byte aligned), and the caller runs
// the generic kernel.
int bb_lift_fast(bb_ctx* ctx, const DegTables* t, int64_t K, int nfaces, const void* x,
                 void* out, cudaStream_t st) {
  if (nfaces == 4 && ((((uintptr_t)x) | ((uintptr_t)out)) & 15) != 0) return -1;
#define BB_LF(n_)                                                                  \
  case n_:                                                                         \
    return nfaces == 4 ? bblift::launch_lift4<n_>(ctx, t, K, x, out, st)                      \
                       : bblift::launch_lift1<n_>(ctx, K, x, out, st);
  switch (t->N) {
    // the single-face kernel stops at N = 12 (its 32-element tiles leave too few warps per SM
    // above); the level-parallel kernel runs it there
    BB_LF(1) BB_LF(2) BB_LF(3) BB_LF(4) BB_LF(5) BB_LF(6) BB_LF(7) BB_LF(8) BB_LF(9)
    BB_LF(10) BB_LF(11) BB_LF(12)
    case 13:
      return nfaces == 4 ? bblift::launch_lift4<13>(ctx, t, K, x, out, st) : -1;
    case 14:
      return nfaces == 4 ? bblift::launch_lift4<14>(ctx, t, K, x, out, st) : -1;
    case 15:
      return nfaces == 4 ? bblift::launch_lift4<15>(ctx, t, K, x, out, st) : -1;
    default:
      return -1;
  }
#undef BB_LF
}
