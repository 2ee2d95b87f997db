// The psi forward kernels, df64, three or four input dimensions (one translation unit per kernel family, precision and
// width, so the build compiles them in parallel).
#include "psi_impl.cuh"

int psi_fwd_df64_q4(const psi_impl::PsiArgs<double>& a, cudaStream_t st) { return psi_impl::launch_fwd_q<df64, 4>(a, st); }

// the translation unit's bounds word (debug build; 0 otherwise)
GPK_BOUNDS_READER(psi_fwd_df64_q4)
