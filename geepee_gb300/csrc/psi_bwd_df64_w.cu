// The psi backward kernels, df64, for three, four and more than five input dimensions (a translation unit
// of their own, so the build compiles them beside the other widths).
#include "psi_impl.cuh"

int psi_bwd_df64_w(const psi_impl::PsiArgs<double>& a, int QC, const psi_impl::BLayout& lo, size_t sm, bool two, cudaStream_t st) {
  return psi_impl::bwd_wide<df64>(a, QC, lo, sm, two, st);
}

// the translation unit's bounds word (debug build; 0 otherwise)
GPK_BOUNDS_READER(psi_bwd_df64_w)
