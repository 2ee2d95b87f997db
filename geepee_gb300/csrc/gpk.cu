// Library-wide host helpers: version, per-thread error text, device properties.
#include <algorithm>

#include "common.cuh"

namespace gpk {
thread_local char g_err[512] = "";

int sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cache[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev] = n;
  }
  return cache[dev];
}
}  // namespace gpk

extern "C" int gpk_version(void) {
  GPK_NVTX("gpk_version"); return 1; }
extern "C" const char* gpk_last_error(void) { return gpk::g_err; }

// the other translation units' bounds words (common.cuh, GPK_BOUNDS_READER)
unsigned gpk_bounds_word_algebra();
unsigned gpk_bounds_word_dense();
unsigned gpk_bounds_word_kern();
unsigned gpk_bounds_word_psi_api();
unsigned gpk_bounds_word_psi_bwd_df64();
unsigned gpk_bounds_word_psi_bwd_f32();
unsigned gpk_bounds_word_psi_fwd_df64_q2();
unsigned gpk_bounds_word_psi_fwd_df64_q4();
unsigned gpk_bounds_word_psi_fwd_df64_q5();
unsigned gpk_bounds_word_psi_bwd_df64_w();
unsigned gpk_bounds_word_psi_fwd_df64_q8();
unsigned gpk_bounds_word_psi_fwd_f32_q2();
unsigned gpk_bounds_word_psi_fwd_f32_q4();
unsigned gpk_bounds_word_psi_fwd_f32_q5();
unsigned gpk_bounds_word_psi_bwd_f32_w();
unsigned gpk_bounds_word_psi_fwd_f32_q8();

extern "C" int gpk_debug_bounds(unsigned int* word) {
  GPK_NVTX("gpk_debug_bounds");
  if (!word) return gpk::fail(GPK_EINVAL, "debug_bounds: null output");
  *word = gpk_bounds_word_algebra() | gpk_bounds_word_dense() | gpk_bounds_word_kern() | gpk_bounds_word_psi_api() |
          gpk_bounds_word_psi_bwd_df64() | gpk_bounds_word_psi_bwd_f32() | gpk_bounds_word_psi_fwd_df64_q2() |
          gpk_bounds_word_psi_fwd_df64_q5() | gpk_bounds_word_psi_fwd_df64_q8() | gpk_bounds_word_psi_fwd_f32_q2() |
          gpk_bounds_word_psi_fwd_f32_q5() | gpk_bounds_word_psi_fwd_f32_q8() | gpk_bounds_word_psi_fwd_df64_q4() |
          gpk_bounds_word_psi_fwd_f32_q4() | gpk_bounds_word_psi_bwd_df64_w() | gpk_bounds_word_psi_bwd_f32_w();
#ifdef GPK_DEBUG_BOUNDS
  return 1;
#else
  return 0;
#endif
}

namespace {

// Eight lanes per output element j: lane l sums the partials c = l, l + 8, ... in order, then
// the eight lane sums combine over a fixed butterfly (both partners compute the same sum, as
// IEEE addition commutes), and lane 0 adds the total into the element's destination.  Plain
// float64 additions: FP64 issues slowly on this GPU, and a compensated sum would cost ~8x
// for ~150 partials whose rounding (~150 ulp at worst) is far below the df64 results' own.
__global__ void __launch_bounds__(256) reduce_partials_kernel(const double* part, int nparts, long stride,
                                                              gpk::RedPlan plan) {
  const long j = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 3;
  const int l = threadIdx.x & 7;
  double s0 = 0.0, s1 = 0.0;   // two chains, joined in a fixed order
  if (j < stride) {
    int k = l;
    for (; k + 8 < nparts; k += 16) {
      s0 += part[(size_t)k * stride + j];
      s1 += part[(size_t)(k + 8) * stride + j];
    }
    if (k < nparts) s0 += part[(size_t)k * stride + j];
  }
  double s = s0 + s1;
#pragma unroll
  for (int m = 1; m < 8; m <<= 1) s = s + __shfl_xor_sync(0xffffffffu, s, m);
  if (l != 0 || j >= stride) return;
  const double v = s;
  long off = 0;
  for (int i = 0; i < plan.nseg; ++i) {
    const gpk::RedSeg& g = plan.seg[i];
    if (j < off + g.len) {
      if (!g.dst) return;
      const long jj = j - off;
      if (g.kind == 0) {
        g.dst[jj] += v;
      } else {
        const long P = (long)g.M * (g.M + 1) / 2;
        const long d = jj / P;
        int a, b;
        tri_pair((int)(jj - d * P), a, b);
        double* m = g.dst + (size_t)d * g.M * g.M;
        m[(size_t)a * g.M + b] += v;
        if (a != b) m[(size_t)b * g.M + a] += v;
      }
      return;
    }
    off += g.len;
  }
}

}  // namespace

namespace gpk {
int reduce_partials(const double* part, int nparts, const RedPlan& plan, cudaStream_t st) {
  const long stride = plan.stride();
  if (stride == 0 || nparts <= 0) return GPK_OK;
  const long threads = stride * 8;
  reduce_partials_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(part, nparts, stride, plan);
  return check_launch("reduce_partials");
}
}  // namespace gpk

// ---- a layer's whole backward in one call ----
namespace {
// the float64 sums of a backward: dsf2 and dl first in the workspace, then (FP32) dZ, dA and dB, which
// in float64 are the caller's tensors themselves
struct LayerSums {
  double *dsf2, *dl, *dZ, *dA, *dB;
  long nZ, nA, nB, used;   // elements; doubles of the workspace taken
};
LayerSums layer_sums(int prec, int M, int Q, int Dout, void* dZ, void* dA, void* dB, double* work) {
  LayerSums s{};
  s.nZ = (long)M * Q;
  s.nA = (long)Dout * M;
  s.nB = (long)Dout * M * M;
  s.dsf2 = work;
  s.dl = work + 1;
  s.used = 1 + Q;
  if (prec == GPK_FP32) {
    s.dZ = work + s.used;
    s.dA = s.dZ + s.nZ;
    s.dB = s.dA + s.nA;
    s.used += s.nZ + s.nA + s.nB;
  } else {
    s.dZ = (double*)dZ;
    s.dA = (double*)dA;
    s.dB = (double*)dB;
  }
  return s;
}
__global__ void __launch_bounds__(256) zero_sums_kernel(LayerSums s, int Q) {
  const long t0 = (long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long)gridDim.x * blockDim.x;
  if (t0 < 1 + Q) s.dsf2[t0] = 0.0;
  for (long i = t0; i < s.nZ; i += nt) s.dZ[i] = 0.0;
  for (long i = t0; i < s.nA; i += nt) s.dA[i] = 0.0;
  for (long i = t0; i < s.nB; i += nt) s.dB[i] = 0.0;
}
int zero_sums(const LayerSums& s, int Q, cudaStream_t st) {
  zero_sums_kernel<<<(int)std::min((s.nB + 255) / 256, 2L * gpk::sm_count()), 256, 0, st>>>(s, Q);
  return gpk::check_launch("layer_bwd");
}
}  // namespace

extern "C" int gpk_psi_layer_bwd(int prec, int N, int M, int Q, int Dout, const void* mu, const void* var,
                                 const void* Z, const double* lls2, const double* lsf2, const void* A, const void* B,
                                 const void* m, const void* dm, const void* dv, void* dZ, void* dA, void* dB,
                                 void* dmu, void* dvar, double* g_l, double* g_s, double* work, long work_elems,
                                 void* stream) {
  GPK_NVTX("gpk_psi_layer_bwd");
  GPK_REQUIRE(prec == GPK_DF64 || prec == GPK_FP32, "psi_layer_bwd: unknown precision %d", prec);
  GPK_REQUIRE(N >= 0 && M >= 1 && Q >= 1 && Dout >= 1, "psi_layer_bwd: bad sizes N=%d M=%d Q=%d Dout=%d", N, M, Q, Dout);
  GPK_REQUIRE(dZ && dA && dB && work, "psi_layer_bwd: null output or workspace");
  const LayerSums s = layer_sums(prec, M, Q, Dout, dZ, dA, dB, work);
  GPK_REQUIRE(work_elems > s.used, "psi_layer_bwd: workspace of %ld doubles, more than %ld needed", work_elems, s.used);
  int rc = zero_sums(s, Q, gpk::as_stream(stream));
  if (rc == GPK_OK)
    rc = gpk_psi_bwd_ws(prec, N, M, Q, Dout, mu, var, Z, lls2, lsf2, A, B, m, dm, dv, nullptr, 0, s.dsf2, s.dl, s.dZ,
                        s.dA, s.dB, dmu, dvar, work + s.used, work_elems - s.used, stream);
  if (rc == GPK_OK)
    rc = gpk::moment_grads(prec, Q, lls2, lsf2, s.dsf2, dv, (long)N * Dout, g_l, g_s, prec == GPK_FP32 ? 3 : 0,
                           {s.nZ, s.nA, s.nB}, {dZ, dA, dB}, stream);
  return rc;
}

extern "C" int gpk_det_layer_bwd(int prec, int N, int M, int D, int Dout, const void* x, int ldx, const void* Z,
                                 const double* lls2, const double* lsf2, const void* A, const void* kfu,
                                 const void* Bk, const void* dm, const void* dv, void* dZ, void* dA, void* dB,
                                 void* dx, double* g_l, double* g_s, double* work, long work_elems, void* stream) {
  GPK_NVTX("gpk_det_layer_bwd");
  GPK_REQUIRE(prec == GPK_DF64 || prec == GPK_FP32, "det_layer_bwd: unknown precision %d", prec);
  GPK_REQUIRE(N >= 0 && M >= 1 && D >= 1 && Dout >= 1, "det_layer_bwd: bad sizes N=%d M=%d D=%d Dout=%d", N, M, D, Dout);
  GPK_REQUIRE(dZ && dA && dB && work, "det_layer_bwd: null output or workspace");
  const LayerSums s = layer_sums(prec, M, D, Dout, dZ, dA, dB, work);
  GPK_REQUIRE(work_elems > s.used, "det_layer_bwd: workspace of %ld doubles, more than %ld needed", work_elems, s.used);
  double* const rest = work + s.used;
  const long nrest = work_elems - s.used;
  int rc = zero_sums(s, D, gpk::as_stream(stream));
  if (rc == GPK_OK)
    rc = gpk_det_bwd_ws(prec, N, M, D, Dout, x, ldx, Z, lls2, lsf2, A, kfu, Bk, dm, dv, nullptr, s.dsf2, s.dl, s.dZ,
                        s.dA, dx, rest, nrest, stream);
  if (rc == GPK_OK) rc = gpk_gram_ws(prec, N, M, Dout, kfu, kfu, dv, s.dB, rest, nrest, stream);
  if (rc == GPK_OK)
    rc = gpk::moment_grads(prec, D, lls2, lsf2, s.dsf2, dv, (long)N * Dout, g_l, g_s, prec == GPK_FP32 ? 3 : 0,
                           {s.nZ, s.nA, s.nB}, {dZ, dA, dB}, stream);
  return rc;
}

extern "C" int gpk_work_elems(int op, int N, int M, int D, int Dout, long* elems) {
  GPK_NVTX("gpk_work_elems");
  GPK_REQUIRE(elems, "work_elems: null output");
  GPK_REQUIRE(N >= 0 && M >= 1 && D >= 1 && Dout >= 1, "work_elems: bad sizes N=%d M=%d D=%d Dout=%d", N, M, D, Dout);
  switch (op) {
    case GPK_OP_PSI_BWD: *elems = psi_bwd_work_elems(M, D, Dout); return GPK_OK;
    case GPK_OP_DET_BWD: *elems = det_bwd_work_elems(N, M, D, Dout); return GPK_OK;
    case GPK_OP_GRAM: *elems = gram_work_elems(N, M, Dout); return GPK_OK;
    case GPK_OP_TRACE_KZZ: *elems = trace_kzz_work_elems(M, D); return GPK_OK;
    default: return gpk::fail(GPK_EINVAL, "work_elems: unknown operation %d", op);
  }
}
