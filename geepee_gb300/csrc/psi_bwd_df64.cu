// df64 instantiation of the psi backward kernels (one translation unit per kernel family
// and precision, so the build compiles them in parallel).
#include "psi_impl.cuh"

int psi_bwd_df64_w(const psi_impl::PsiArgs<double>& a, int QC, const psi_impl::BLayout& lo, size_t sm, bool two, cudaStream_t st);
int psi_bwd_df64(const psi_impl::PsiArgs<double>& a, cudaStream_t st) { return psi_impl::launch_bwd<df64>(a, psi_bwd_df64_w, st); }

// the translation unit's bounds word (debug build; 0 otherwise)
GPK_BOUNDS_READER(psi_bwd_df64)
