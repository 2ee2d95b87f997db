// ARD exponentiated-quadratic kernel matrices and the deterministic-input sparse-GP
// layer (first DGP layer / SGPR): fused forward contractions and the per-row backward.
#include "common.cuh"

namespace {

constexpr int DMAXK = 64;   // max input dimension
constexpr int DO_MAX = 4;   // max output dimension of a layer

template <typename T>
struct Hyp {
  T inv_l2[DMAXK];   // 1/ell^2
  T lsf;             // log sf^2
  T sf2;
};

template <typename T>
__device__ void load_hyp(Hyp<T>& h, const double* lls2, const double* lsf2, int D, const float2* tab) {
  typedef typename Num<T>::store_t S;
  for (int d = threadIdx.x; d < D; d += blockDim.x)
    h.inv_l2[d] = exp_tab(neg(Num<T>::ld(static_cast<S>(lls2[d]))), tab);
  if (threadIdx.x == 0) {
    h.lsf = Num<T>::ld(static_cast<S>(lsf2[0]));
    h.sf2 = exp_tab(h.lsf, tab);
  }
}

// K[n,m] = exp(lsf - 1/2 sum_d (x-z)^2 / l_d) (+ jitter on the diagonal): FP32, and matrices with a jitter.  A CTA takes KR rows
// and KC columns: those rows of x and columns' Z arrive in shared memory by asynchronous copies,
// then 256 threads sweep the KR x KC block.
constexpr int KR = 8, KC = 128;
template <typename T>
__global__ void __launch_bounds__(256) kern_matrix_kernel(int N, int M, int D, const typename Num<T>::store_t* x,
                                                          int ldx, const typename Num<T>::store_t* z, int ldz,
                                                          const double* lls2, const double* lsf2, double jitter,
                                                          typename Num<T>::store_t* K, int ldk) {
  typedef typename Num<T>::store_t S;
  extern __shared__ __align__(16) char smem_raw[];
  float2* tab = reinterpret_cast<float2*>(smem_raw);
  Hyp<T>* h = reinterpret_cast<Hyp<T>*>(smem_raw + 256 * sizeof(float2));
  T* xs = reinterpret_cast<T*>(smem_raw + 256 * sizeof(float2) + sizeof(Hyp<T>));   // [KR][D]
  T* zs = xs + KR * D;                                                                  // [KC][D]
  const int tid = threadIdx.x;
  const int m0 = blockIdx.x * KC, n0 = blockIdx.y * KR;
  const int nr = min(KR, N - n0), nc = min(KC, M - m0);
  for (int e = tid; e < nr * D; e += 256) {
    const int r = e / D, d = e - r * D;
    async_copy(reinterpret_cast<S*>(xs) + e, x + (size_t)(n0 + r) * ldx + d);
  }
  for (int e = tid; e < nc * D; e += 256) {
    const int c = e / D, d = e - c * D;
    async_copy(reinterpret_cast<S*>(zs) + e, z + (size_t)(m0 + c) * ldz + d);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  load_exp_table(tab);
  __syncthreads();
  convert_in_place(xs, (long)nr * D, tid, 256);
  convert_in_place(zs, (long)nc * D, tid, 256);
  load_hyp(*h, lls2, lsf2, D, tab);
  __syncthreads();
  for (int e = tid; e < nr * nc; e += 256) {
    const int r = e / nc, c = e - r * nc;
    const int n = n0 + r, m = m0 + c;
    T rr = Num<T>::zero();
    for (int d = 0; d < D; ++d) {
      const T df = sub(xs[r * D + d], zs[c * D + d]);
      rr = fma_(mul(df, df), h->inv_l2[d], rr);
    }
    T k = exp_tab(sub(h->lsf, scale2(rr, -1)), tab);
    if (jitter != 0.0 && n == m) k = add(k, Num<T>::ld(static_cast<S>(jitter)));
    K[(size_t)n * ldk + m] = Num<T>::st(k);
  }
}

// ---- the kernel matrix in double-float precision, exponents in fixed point ----
// log2 K[n,m] = log2 sf^2 - sum_d (x'_nd - z'_md)^2 with the coordinates x' = x sqrt(log2(e)/2) / ell
// as two words, high 2^-26 + low 2^-57: a difference is two integer subtractions, exact, and its
// square two 32 x 32 -> 64-bit multiply-adds (the low word's square, at most 2^-52, is left out), where
// the double-float difference, square and scaling take 32 instructions; the exponential then comes from
// the exponent's bits (exp2_fx).  High words and sums are taken modulo 2^32 and 2^64, so that only differences
// need the range: a float sum of the squares, of coordinates about the first pseudo-input's, says which are
// meant.  At 256 or more the entry is zero (below 2^-126 with sf^2 < 2^126), below it no difference and no
// sum leaves the range.  The floats are good to 2^-6 up to 2^16 lengthscales from that pseudo-input;
// farther pseudo-inputs, and inputs that are not finite, have NaN for theirs, which sends the entries they
// meet to the double-float form (ard_general); farther inputs meet no nearer pseudo-input.  Coordinates by
// their distance from the origin instead took that form beyond 18.8 lengthscales of it, an entry at a time: 109 us
// at N = 20000, M = 100, D = 8, inputs about 37 lengthscales off, where this takes 27.
struct __align__(16) ArdHyp {
  unsigned long long ms[DMAXK];   // sqrt(log2(e)/2) / ell_d: its significand,
  int sh[DMAXK];        // 2093 less its exponent field (ard_coord)
  float s[DMAXK];       // and its float (NaN out of range: every entry takes the general form)
  float2 o[DMAXK];      // the first pseudo-input
  df64 inv_l2[DMAXK];   // 1/ell_d^2 (general form)
  df64 lsf;
  long long c0;         // log2 sf^2 in units of 2^-52, plus exp2_fx's half step
  int flag;             // sf^2 outside the fixed-point range: every entry takes the general form
};
__device__ __forceinline__ void load_ard(ArdHyp& h, const double* lls2, const double* lsf2, int D, const double* z,
                                         ExpTab tab) {
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const double l = lls2[d];
    const double s = exp(-0.5 * l) * 0.84932180028801904272;   // (in float64: its error counts twice the exponent)
    const long long b = __double_as_longlong(s);
    h.ms[d] = ((unsigned long long)b & 0xfffffffffffffULL) | 0x10000000000000ULL;
    h.sh[d] = 2093 - (int)(b >> 52);
    h.s[d] = s > 1e-30 && s < 1e30 ? (float)s : __int_as_float(0x7fffffff);
    const df64 o = fabs(z[d]) < 1e30 ? df_from_double(z[d]) : make_df(0.f);
    h.o[d] = make_float2(o.hi, o.lo);
    h.inv_l2[d] = exp_tab(df_from_double(-l), tab);
  }
  if (threadIdx.x == 32) {
    h.lsf = df_from_double(lsf2[0]);
    const double c = lsf2[0] * 1.4426950408889634074;
    h.flag = !(fabs(c) < 126.0);
    h.c0 = (h.flag ? 0LL : __double2ll_rn(c * 4503599627370496.0)) + kFxHalf;
  }
}
// coordinate x of dimension d times the scale in fixed point: (low, high modulo 2^32, float beside the first
// pseudo-input's, -).  The product of the two 53-bit significands is exact, its bits below 2^-57 cut off; on
// the integer pipes, because a product and its rounding error by the FP64 pipe made the kernel 8% slower.  The
// pseudo-inputs' floats end at 2^16 (ZED).
template <bool ZED>
__device__ __forceinline__ int4 ard_coord(double x, const ArdHyp& h, int d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)(b >> 52) & 0x7ff, sh = h.sh[d] - ex;
  const unsigned long long m = (b & 0xfffffffffffffULL) | 0x10000000000000ULL;
  const unsigned long long lo = m * h.ms[d], hi = __umul64hi(m, h.ms[d]);   // |x| s = (hi : lo) 2^-(57 + sh)
  unsigned long long u = 0;
  if (sh >= 64) u = hi >> min(sh - 64, 63);   // (hi < 2^42)
  else if (sh > 0) u = (lo >> sh) | (hi << (64 - sh));
  else if (sh > -64) u = lo << -sh;
  const long long t = ((long long)b < 0 ? -(long long)u : (long long)u) + (1LL << 30);
  int f = 0x7fffffff;   // not finite
  if (ex < 1150) {
    const df64 v = df_from_double(x);
    f = __float_as_int(__fmul_rn(__fadd_rn(__fsub_rn(v.hi, h.o[d].x), __fsub_rn(v.lo, h.o[d].y)), h.s[d]));
  } else if (ex < 2047) {
    f = 0x7f800000 | (int)(b >> 32 & 0x80000000u);   // beyond the float range
  }
  if (ZED && (f & 0x7fffffff) > 0x47800000) f = 0x7fffffff;
  return make_int4((int)((unsigned)t & 0x7fffffffu) - (1 << 30), (int)(t >> 31), f, 0);
}
__device__ __forceinline__ int4 lds_i4(saddr a) {
  int4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
// the exponents X and float sums of squares f of R rows against one column, D coordinates each:
// x + i * xstep (row i) and z
template <int R>
__device__ __forceinline__ void ard_exponents(saddr x, saddr xstep, saddr z, int D, long long c0, long long (&X)[R],
                                              float (&f)[R]) {
  long long mid[R];
#pragma unroll
  for (int i = 0; i < R; ++i) X[i] = c0, f[i] = 0.f;
  // the cross terms of 16 dimensions stay below 2^63: sum h^2 < 2^60 where the entry is not zero, |l| < 2^31
  for (int d0 = 0; d0 < D; d0 += 16) {
    const int dn = min(16, D - d0);
#pragma unroll
    for (int i = 0; i < R; ++i) mid[i] = 0;
#pragma unroll 4
    for (int d = 0; d < dn; ++d) {
      const int4 zd = lds_i4(z);
      z += 16;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int4 xd = lds_i4(x + i * xstep);
        const int h = xd.y - zd.y, l = xd.x - zd.x;
        const float t = __int_as_float(xd.z) - __int_as_float(zd.z);
        X[i] = mad_wide(-h, h, X[i]);
        mid[i] = mad_wide(h, l, mid[i]);
        f[i] = __fmaf_rn(t, t, f[i]);
      }
      x += 16;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) X[i] -= mid[i] >> 30;
  }
}
__device__ __noinline__ df64 ard_general(const double* x, const double* z, int D, const ArdHyp& h, const float2* tab) {
  df64 rr = make_df(0.f);
  for (int d = 0; d < D; ++d) {
    const double diff = x[d] - z[d];   // (far from the origin a coordinate's own 48 bits are too few)
    if (fabs(diff) < 1.7e308 && fabs(diff) * (double)h.s[d] > 1048576.0) return make_df(0.f);
    const df64 df = df_from_double(diff);
    rr = fma_(mul(df, df), h.inv_l2[d], rr);
  }
  return exp_tab(sub(h.lsf, scale2(rr, -1)), ExpTab{tab});
}

// K (float64): a CTA takes FC columns and row tiles of FR; a thread one column and FR / (256 / FC) rows,
// four at a time, so that a column's coordinate is loaded once for four rows.  As many CTAs as
// are resident at once share the tiles: the tables and the columns are staged once a CTA.
// Bound by the integer and FP32 pipes: 20000 x 100, D = 8 in 27 us (49 before), 20000 x 200, D = 16 in
// 67 us (256 before).
constexpr int FR = 16, FC = 128, FCTA = 3;
__global__ void __launch_bounds__(256, FCTA) kern_fx_kernel(int N, int M, int D, const double* x, int ldx,
                                                            const double* z, int ldz, const double* lls2,
                                                            const double* lsf2, double* K, int ldk) {
  extern __shared__ __align__(16) char smem_raw[];
  float2* tab = reinterpret_cast<float2*>(smem_raw);
  ArdHyp* h = reinterpret_cast<ArdHyp*>(smem_raw + kFxTab * sizeof(float2));
  int4* xs = reinterpret_cast<int4*>(h + 1);             // [2][FR][D]: this tile's and the next one's
  const int DZ = D | 1;                                  // (odd: the columns' banks differ)
  int4* zs = xs + 2 * FR * D;                            // [FC][DZ]
  const int tid = threadIdx.x;
  const int nmb = (M + FC - 1) / FC, m0 = (int)(blockIdx.x % nmb) * FC, nc = min(FC, M - m0);
  const int ntile = (N + FR - 1) / FR, step = (int)(gridDim.x / nmb);
  load_exp2_table(tab);
  __syncthreads();
  load_ard(*h, lls2, lsf2, D, z, ExpTab{tab});
  __syncthreads();
  auto rows = [&](int tile, int b) {
    const int n0 = tile * FR, nr = min(FR, N - n0);
    for (int e = tid; e < nr * D; e += 256) {
      const int r = e / D, d = e - r * D;
      xs[b * FR * D + e] = ard_coord<false>(x[(size_t)(n0 + r) * ldx + d], *h, d);
    }
  };
  for (int e = tid; e < nc * D; e += 256) {
    const int c = e / D, d = e - c * D;
    zs[c * DZ + d] = ard_coord<true>(z[(size_t)(m0 + c) * ldz + d], *h, d);
  }
  rows((int)(blockIdx.x / nmb), 0);
  __syncthreads();
  const int c = tid & (FC - 1), m = m0 + c;
  const saddr at = sm_addr(tab), az = sm_addr(zs + c * DZ);
  const bool hf = h->flag;
  int b = 0;
  for (int tile = (int)(blockIdx.x / nmb); tile < ntile; tile += step, b ^= 1) {
    const int n0 = tile * FR, nr = min(FR, N - n0);
    if (tile + step < ntile) rows(tile + step, b ^ 1);
    if (c < nc) {
      for (int r0 = (tid >> 7) * 4; r0 < nr; r0 += 8) {
        long long X[4];
        float f[4];
        // rows past nr read the tile's stale coordinates; their entries are not stored
        ard_exponents<4>(sm_addr(xs + (b * FR + r0) * D), D * 16, az, D, h->c0, X, f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = n0 + r0 + i;
          if (r0 + i < nr) {
            double k = exp2_fx_double<-1022>(X[i], at);
            if (!(f[i] < 256.f) || hf)
              k = f[i] >= 256.f && !hf ? 0.0
                                       : df_to_double(ard_general(x + (size_t)n * ldx, z + (size_t)m * ldz, D, *h, tab));
            K[(size_t)n * ldk + m] = k;
          }
        }
      }
    }
    __syncthreads();
  }
}

// Deterministic-input layer forward for rows n:
//   k_n = K(x_n, Z);  m_nd = k_n . A_d;  Bk_ndb = sum_a B_d[a,b] k_na;  v_nd = sf2 + k_n . Bk_nd
// (geepee/aep_models.py:142-158, base_models.py:265-284).
//
// A CTA takes tiles of FT rows for one output d (blockIdx.y).  The rows' kernel values go to
// shared memory; then, for each block of 128 columns b, every thread owns one column and FT/2
// rows of Bk and
// runs their sums over a from shared memory, while B_d streams through shared memory in
// chunks of FKA rows.  The next chunk's global loads are issued before the current chunk is
// used (register double buffer), so the stream costs one memory latency per tile, not one
// per chunk.  m and v are reduced over the columns by warp shuffles.
constexpr int FT = 8;      // rows per tile
constexpr int FKA = 32;    // rows of B_d per staged chunk
constexpr int FCB = 128;   // columns per block
constexpr int FNL = FKA * FCB / 256;   // staged elements per thread per chunk
template <typename T>
__global__ void __launch_bounds__(256) det_fwd_kernel(int N, int M, int D, int Dout,
                                                      const typename Num<T>::store_t* x, int ldx,
                                                      const typename Num<T>::store_t* z, const double* lls2,
                                                      const double* lsf2, const typename Num<T>::store_t* A,
                                                      const typename Num<T>::store_t* B,
                                                      typename Num<T>::store_t* kfu,
                                                      typename Num<T>::store_t* Bk,
                                                      typename Num<T>::store_t* m_out,
                                                      typename Num<T>::store_t* v_out, int zstage) {
  typedef typename Num<T>::store_t S;
  extern __shared__ __align__(16) char smem_raw[];
  float2* tab = reinterpret_cast<float2*>(smem_raw);
  Hyp<T>* h = reinterpret_cast<Hyp<T>*>(smem_raw + 256 * sizeof(float2));
  T* kr = reinterpret_cast<T*>(smem_raw + 256 * sizeof(float2) + sizeof(Hyp<T>));   // [FT][M]
  T* Bc = kr + FT * M;                       // [FKA][FCB]
  T* red = Bc + FKA * FCB;                   // [8 warps][DO_MAX][FT/2][2]
  T* xs = red + 8 * DO_MAX * FT;             // [FT][D]
  T* zs = xs + FT * D;                       // [M][D] when staged
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = tid & (FCB - 1), rh = tid >> 7;   // column in the block, row half
  load_exp_table(tab);
  if (zstage)
    for (int i = tid; i < M * D; i += 256) zs[i] = Num<T>::ld(z[i]);
  __syncthreads();
  load_hyp(*h, lls2, lsf2, D, tab);
  const int d = blockIdx.y;   // this CTA's output
  const int nca = (M + FKA - 1) / FKA, ncb = (M + FCB - 1) / FCB, nq = ncb * nca;
  const size_t MM = (size_t)M * M;
  auto issue = [&](int q, S* raw) {
    const int cb0 = (q / nca) * FCB, a0 = (q % nca) * FKA;
    const S* Bd = B + (size_t)d * MM;
#pragma unroll
    for (int u = 0; u < FNL; ++u) {
      const int e = tid + u * 256, aa = e / FCB, cc = e % FCB;
      const int a = a0 + aa, b = cb0 + cc;
      raw[u] = (a < M && b < M) ? Bd[(size_t)a * M + b] : S(0);
    }
  };
  for (int n0 = blockIdx.x * FT; n0 < N; n0 += gridDim.x * FT) {
    S raw[FNL];
    issue(0, raw);   // the first chunk's loads overlap the kernel values below
    for (int i = tid; i < FT * D; i += 256) {
      const int r = i / D, q = i - r * D, n = n0 + r;
      xs[i] = n < N ? Num<T>::ld(x[(size_t)n * ldx + q]) : Num<T>::zero();
    }
    __syncthreads();
    for (int i = tid; i < FT * M; i += 256) {
      const int r = i / M, mm = i - r * M, n = n0 + r;
      T k = Num<T>::zero();
      if (n < N) {
        T rr = Num<T>::zero();
        for (int q = 0; q < D; ++q) {
          const T zq = zstage ? zs[mm * D + q] : Num<T>::ld(z[(size_t)mm * D + q]);
          const T df = sub(xs[r * D + q], zq);
          rr = fma_(mul(df, df), h->inv_l2[q], rr);
        }
        k = exp_tab(sub(h->lsf, scale2(rr, -1)), tab);
        if (kfu && d == 0) kfu[(size_t)n * M + mm] = Num<T>::st(k);
      }
      kr[i] = k;
    }
    T acc[FT / 2], pm[FT / 2], pv[FT / 2];
    for (int q = 0; q < nq; ++q) {
      const int cbi = q / nca, ai = q % nca;
      const int a0 = ai * FKA, b = cbi * FCB + col;
      __syncthreads();   // the previous chunk is consumed (and kr is complete)
#pragma unroll
      for (int u = 0; u < FNL; ++u) Bc[tid + u * 256] = Num<T>::ld(raw[u]);
      __syncthreads();
      if (q + 1 < nq) issue(q + 1, raw);
      if (q == 0) {
#pragma unroll
        for (int r = 0; r < FT / 2; ++r) pm[r] = pv[r] = Num<T>::zero();
      }
      if (ai == 0) {
#pragma unroll
        for (int r = 0; r < FT / 2; ++r) acc[r] = Num<T>::zero();
      }
      const int ka = min(FKA, M - a0);
      const T* kt = kr + (rh * (FT / 2)) * M + a0;
#pragma unroll 4
      for (int aa = 0; aa < ka; ++aa) {
        const T bab = Bc[aa * FCB + col];
#pragma unroll
        for (int r = 0; r < FT / 2; ++r) acc[r] = fma_(bab, kt[r * M + aa], acc[r]);
      }
      if (ai == nca - 1 && b < M) {
        const T ad = Num<T>::ld(A[(size_t)d * M + b]);
#pragma unroll
        for (int r = 0; r < FT / 2; ++r) {
          const int rl = rh * (FT / 2) + r, n = n0 + rl;
          if (n < N && Bk) Bk[((size_t)n * Dout + d) * M + b] = Num<T>::st(acc[r]);
          const T kb = kr[rl * M + b];
          pm[r] = fma_(kb, ad, pm[r]);
          pv[r] = fma_(kb, acc[r], pv[r]);
        }
      }
      if (ai == nca - 1 && cbi == ncb - 1) {
#pragma unroll
        for (int r = 0; r < FT / 2; ++r) {
          const T sm = warp_sum(pm[r]), sv = warp_sum(pv[r]);
          if (lane == 0) {
            red[((warp * DO_MAX + d) * (FT / 2) + r) * 2] = sm;
            red[((warp * DO_MAX + d) * (FT / 2) + r) * 2 + 1] = sv;
          }
        }
      }
    }
    __syncthreads();
    for (int rl = tid; rl < FT; rl += 256) {
      const int n = n0 + rl;
      const int hh = rl / (FT / 2), r = rl - hh * (FT / 2);
      if (n < N) {
        T mm = Num<T>::zero(), vv = Num<T>::zero();
#pragma unroll
        for (int w = 0; w < 4; ++w) {   // the four warps of row half hh
          const int ww = hh * 4 + w;
          mm = add(mm, red[((ww * DO_MAX + d) * (FT / 2) + r) * 2]);
          vv = add(vv, red[((ww * DO_MAX + d) * (FT / 2) + r) * 2 + 1]);
        }
        if (m_out) m_out[(size_t)n * Dout + d] = Num<T>::st(mm);
        if (v_out) v_out[(size_t)n * Dout + d] = Num<T>::st(add(h->sf2, vv));
      }
    }
  }
}

// The deterministic-input layer's contractions from given kernel values kfu [N,M]:
//   m_nd = kfu_n . A_d;  Bk_ndb = sum_a B_d[a,b] kfu_na;  v_nd = sf2 + kfu_n . Bk_nd
// (geepee/aep_models.py:142-158 once Kfu is formed).  A CTA takes CR rows; warp w works on row
// w % CR and column half w / CR, lane l on columns b = 64 h + l + 32 j (j < 2), for all DB
// outputs, so each thread runs 2 DB independent sums over a.  All of B (Dout M^2) and the CTA's
// kernel rows sit in shared memory (asynchronous copies, converted in place);
// m and v are warp sums, then the two halves'
// sums are added in a fixed order.
constexpr int CR = 8;              // rows per CTA
constexpr int CT = CR * 2 * 32;    // threads: (row, column half) per warp
template <typename T, int DB>
__global__ void __launch_bounds__(CT) det_contract_kernel(int N, int M, int Dout,
                                                          const typename Num<T>::store_t* kfu,
                                                          const double* lsf2,
                                                          const typename Num<T>::store_t* A,
                                                          const typename Num<T>::store_t* B,
                                                          typename Num<T>::store_t* Bk,
                                                          typename Num<T>::store_t* m_out,
                                                          typename Num<T>::store_t* v_out) {
  typedef typename Num<T>::store_t S;
  extern __shared__ __align__(16) char smem_raw[];
  float2* tab = reinterpret_cast<float2*>(smem_raw);
  T* Bs = reinterpret_cast<T*>(smem_raw + 256 * sizeof(float2));   // [Dout][M][M]
  T* kr = Bs + (size_t)Dout * M * M;                                 // [CR][M]
  T* red = kr + (size_t)CR * M;                                      // [2][CR][DB][2] half sums
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int r = w % CR, h = w / CR;
  const int n0 = blockIdx.x * CR, n = n0 + r;
  const int nB = Dout * M * M, nr = min(CR, N - n0);
  stage_async(reinterpret_cast<S*>(Bs), B, nB, tid, CT);
  stage_async(reinterpret_cast<S*>(kr), kfu + (size_t)n0 * M, (long)nr * M, tid, CT);
  load_exp_table(tab);
  __syncthreads();
  convert_in_place(Bs, nB, tid, CT);
  convert_in_place(kr, (long)nr * M, tid, CT);
  __syncthreads();
  const bool live = n < N;   // warp-uniform; a dead row still reaches the barrier below
  const T* k = kr + (size_t)(live ? r : 0) * M;
  // columns past M read the row's last column (in bounds) and are never stored
  const int c0 = min(64 * h + lane, M - 1), c1 = min(64 * h + lane + 32, M - 1);
  T acc[DB][2];
#pragma unroll
  for (int d = 0; d < DB; ++d) acc[d][0] = acc[d][1] = Num<T>::zero();
  // output d's columns of B; outputs past Dout (DB = 4 for Dout = 3) read output 0's, in
  // bounds, and are never stored
  const T* B0[DB];
  const T* B1[DB];
#pragma unroll
  for (int d = 0; d < DB; ++d) {
    const size_t off = (size_t)(d < Dout ? d : 0) * M * M;
    B0[d] = Bs + off + c0;
    B1[d] = Bs + off + c1;
  }
  for (int a = 0; a < M; ++a) {
    const T ka = k[a];
    const size_t ra = (size_t)a * M;
#pragma unroll
    for (int d = 0; d < DB; ++d) {
      // det_fwd's operand order, so that the sums match its arithmetic
      acc[d][0] = fma_(B0[d][ra], ka, acc[d][0]);
      acc[d][1] = fma_(B1[d][ra], ka, acc[d][1]);
    }
  }
  T pm[DB], pv[DB];
#pragma unroll
  for (int d = 0; d < DB; ++d) {
    pm[d] = pv[d] = Num<T>::zero();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int b = 64 * h + lane + 32 * j;
      if (live && b < M && d < Dout) {
        if (Bk) Bk[((size_t)n * Dout + d) * M + b] = Num<T>::st(acc[d][j]);
        pm[d] = fma_(k[b], Num<T>::ld(A[(size_t)d * M + b]), pm[d]);
        pv[d] = fma_(k[b], acc[d][j], pv[d]);
      }
    }
    pm[d] = warp_sum(pm[d]);
    pv[d] = warp_sum(pv[d]);
    if (lane == 0) {
      red[((h * CR + r) * DB + d) * 2] = pm[d];
      red[((h * CR + r) * DB + d) * 2 + 1] = pv[d];
    }
  }
  __syncthreads();
  if (h == 0 && lane == 0 && live) {
    const T sf2 = exp_tab(Num<T>::ld(static_cast<S>(lsf2[0])), tab);
#pragma unroll
    for (int d = 0; d < DB; ++d) {
      if (d < Dout) {
        const T mm = add(red[((0 * CR + r) * DB + d) * 2], red[((1 * CR + r) * DB + d) * 2]);
        const T vv = add(red[((0 * CR + r) * DB + d) * 2 + 1], red[((1 * CR + r) * DB + d) * 2 + 1]);
        if (m_out) m_out[(size_t)n * Dout + d] = Num<T>::st(mm);
        if (v_out) v_out[(size_t)n * Dout + d] = Num<T>::st(add(sf2, vv));
      }
    }
  }
}

size_t det_contract_smem(int M, int Dout, size_t tsz) {
  return 256 * sizeof(float2) + ((size_t)Dout * M * M + (size_t)CR * M + 2 * CR * DO_MAX * 2) * tsz;
}

// ---- the deterministic layer's contraction in double-float precision on the tensor cores ----
// For rows n and one output d:  Bk_nb = sum_a B[a,b] k_na,  m_n = k_n . A,  v_n = sf2 + k_n . Bk_n, from
// the kernel rows k.  Bk by digits: B is balanced by powers of two along both indices, B'_ab = B_ab 2^-(r_a + c_b)
// with c_b the largest exponent of column b and r_a <= 0 that of row a beside the c_b, so that every row and
// every column of B' has its largest entry next to 1; the r_a go over to the rows, k'_a = k_a 2^r_a.  Each row of
// k' is scaled by its largest entry; the numbers, below 1/2 then, are taken to 53 bits below the point (k rounded;
// B through its double-float form, ~2^-49 of an entry, truncated), the integer is cut into six balanced digits
// of nine bits (each an exact f16), and a product of two such numbers is the digit products of levels
// i + j <= 6: 26 f16 multiply-adds into f32.  Digit products are at most 2^16, so an accumulator that takes
// at most two of them over 128 terms holds an integer of at most 2^24: the sums of levels 0 to 4 are exact
// (nine accumulators; a longer contraction is folded into 64-bit integers every 128 terms).  Levels 5
// and 6 have one accumulator each, whose last place is below 2^-56 of the largest product.
// Errors: Bk_nb is off by a few 2^-52 of max_a k'_a 2^c_b times sqrt(M), where a double-float sum (14 instructions
// a term, every term rounded) is off by some 2^-48 of sum_a |k_a B_ab|.  Some column b of every row has a sum
// as large as max_a k'_a 2^c_b, so a row of Bk keeps the double-float accuracy relative to its largest
// sums; an entry whose terms are all far smaller keeps it relative to those, not to itself.  m and v keep the
// double-float accuracy relative to their sums of |terms|: A is column M of B' (its own scale, beside the r_a), and
// the sums of |k'_a B'_ab| are estimated from the first digits by one more product.  Where m's is below 1/16 of its
// scales, or sum_b |k_b| 2^c_b sum_a |k'_a B'_ab| below 1/16 of max_a k'_a sum_b |k_b| 2^c_b (few rows: none in the
// deep GP's and the regressions' layers), the row's m, or its v and Bk, are formed again in double-float.
// A CTA of 16 warps takes R = 16 nrt rows at a time, B's digits resident in shared memory in the order
// of the matrix instruction's fragments (restaged by column blocks per row chunk when they do not fit);
// a warp takes 16 x 8 results at a time.  v is summed in an order that depends on M alone, so a row's
// results are the same in any batch.
// One-off staging of B (~12 us at M = 100, 3 of them the balance), then per 32 rows ~5500 cycles of digits, ~17000
// of products (the matrix pipe itself ~10000) and ~7000 of epilogue.  With the rows' kernel launch before it,
// N = 20000, M = 100, two outputs take 181 us (in double-float 752; scaled by the rows' and columns'
// largest entries alone, without the balance and the estimate, 168); N = 777, M = 200 75 us (159; 70); the
// contraction alone at N = 1000, M = 100 22 us (27; 19).
constexpr int DM_T = 512, DM_W = DM_T / 32, DM_S = 6;
// an integer (|x| < 2^61) times 2^-F as a double-float
__device__ __forceinline__ df64 df_of_int(long long x, int F) {
  const float h = (float)(int)(x >> 38), m = (float)(int)((x >> 16) & 0x3fffff), l = (float)(int)(x & 0xffff);
  const df64 a = two_sum(__fmul_rn(h, 4194304.f), m);   // all three are exact; units of 2^16
  return scale2(scale2(add(a, __fmul_rn(l, 1.52587890625e-05f)), 8), 8 - F);
}
// a float in units of 2^-F, truncated (the exponent field at most 189 - F)
__device__ __forceinline__ long long fx_bits_by(float x, int F) {
  const unsigned b = __float_as_uint(x);
  const int e = (int)((b >> 23) & 0xffu), s = e == 0 ? 63 : min(189 - F - e, 63);
  const long long v = (long long)(((unsigned long long)(((b & 0x7fffffu) | 0x800000u) << 7) << 32) >> s);
  return (int)b < 0 ? -v : v;
}
// v 2^(-1 - ex) (|v| < 2^ex), less than 1/2 in magnitude, in units of 2^-53, rounded
__device__ __forceinline__ long long digits_of(double v, int ex) {
  const long long b = __double_as_longlong(v);
  const int be = (int)((b >> 52) & 0x7ff), sh = 1023 + ex - be;   // at least 1
  const long long w = (b & 0xfffffffffffffLL) | 0x10000000000000LL;
  const long long x = sh > 60 || be == 0 ? 0 : (w + (1LL << (sh - 1))) >> sh;
  return b < 0 ? -x : x;
}
// two numbers' digits (|t| <= 2^52, units of 2^-53, t0 in the low half), most significant first
__device__ __forceinline__ void digit_pairs(long long t0, long long t1, unsigned (&w)[DM_S]) {
  const long long bias = 256LL * (1 + (1LL << 9) + (1LL << 18) + (1LL << 27) + (1LL << 36) + (1LL << 45));
  t0 += bias;
  t1 += bias;
  const unsigned l0 = (unsigned)t0 & 0x7ffffffu, l1 = (unsigned)t1 & 0x7ffffffu;
  const unsigned h0 = (unsigned)(t0 >> 27), h1 = (unsigned)(t1 >> 27);
#pragma unroll
  for (int j = 0; j < DM_S; ++j) {
    const unsigned a = j < 3 ? h0 : l0, b = j < 3 ? h1 : l1;
    const int sh = 9 * (2 - j % 3);
    unsigned e = ((a >> sh) & 511u) | ((b >> sh) & 511u) << 16 | 0x64006400u;   // halves 1024 + digit + 256
    asm("sub.rn.f16x2 %0, %0, %1;" : "+r"(e) : "r"(0x65006500u));               // minus 1280
    w[j] = e;
  }
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint4 a, const uint2 b) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y));
}
// the accumulator of digits i of the left and j of the right operand
constexpr int DM_ACC = 11;
__host__ __device__ constexpr int dm_acc(int i, int j) {
  const int base[7] = {0, 1, 2, 4, 6, 9, 10};
  return base[i + j] + (i + j < 5 ? i / 2 : 0);
}
// the accumulators' value of result j, in units of 2^-52 of the scaled operands' product in units of 2^-106
__device__ __forceinline__ long long dm_fold(const float (&acc)[DM_ACC][4], int j) {
  auto S = [&](int i) { return __float2int_rn(acc[i][j]); };
  const int s6 = __float2int_rn(__fmul_rn(acc[10][j], 1.f / 512));
  const long long X = mad_wide(S(0), 1 << 18, mad_wide(S(1), 1 << 9, (long long)(S(2) + S(3))));
  const long long Y = mad_wide(S(4) + S(5), 1 << 18, mad_wide(S(6) + S(7) + S(8), 1 << 9, (long long)(S(9) + s6)));
  return (X << 20) + (Y >> 7);
}
constexpr unsigned POS2 = 0x7fff7fffu;   // the magnitudes of two f16
// one k step: all digit products of a row fragment and a column fragment (strides in fragments), and into mag the
// product of the first digits' magnitudes, of the columns' alone unless BOTH: the sum of magnitudes for rows
// without negative entries (kernel values), never more than it
template <bool BOTH>
__device__ __forceinline__ void dm_step(float (&acc)[DM_ACC][4], float (&mag)[4], const uint4* fa, int sa, const uint2* fb,
                                        int sb) {
  uint4 va[DM_S];
#pragma unroll
  for (int i = 0; i < DM_S; ++i) va[i] = fa[(size_t)i * sa];
#pragma unroll
  for (int j = 0; j < DM_S; ++j) {
    const uint2 vb = fb[(size_t)j * sb];
    if (j == 0) {
      const uint4 a = BOTH ? make_uint4(va[0].x & POS2, va[0].y & POS2, va[0].z & POS2, va[0].w & POS2) : va[0];
      mma_f16(mag, a, make_uint2(vb.x & POS2, vb.y & POS2));
    }
#pragma unroll
    for (int i = 0; i < DM_S; ++i)
      if (i + j <= 6) mma_f16(acc[dm_acc(i, j)], va[i], vb);
  }
}
struct DmSmem {
  unsigned *B, *A;      // digit pairs: [digit][column tile][k step][lane][2], [digit][row tile][k step][lane][4]
  df64 *k, *vp, *v;     // [R][M|1] the rows, [R][NT] parts of v, [R] v
  float2* tp;           // [R][NT] sum_b |k_b| 2^c_b times the first digits' sum of |k'_a B'_ab|, by lanes
  float *t, *e;         // [R] the sum of those; sum_b |k_b| 2^c_b, or -1 where no entry is in the float range
  float* cw;            // [M] 2^(c_b - the largest); 0: a column with a non-finite entry
  int *rexp, *mgen;     // [R] exponent of the scaled row; whether its m takes the double-float form
  int *c, *r;           // [M + 1] exponents c_b (M: A's), [M] r_a
};
__host__ __device__ inline size_t dm_carve(DmSmem* out, char* base, int M, int NB, int R) {
  DmSmem s;
  size_t o = 0;
  auto take = [&](size_t n) {
    char* p = base + o;
    o += (n + 15) & ~(size_t)15;
    return p;
  };
  const int KP = (M + 15) & ~15;
  s.B = (unsigned*)take((size_t)DM_S * NB * KP * 2);
  s.A = (unsigned*)take((size_t)DM_S * R * KP * 2);
  s.k = (df64*)take((size_t)R * (M | 1) * 8);
  s.vp = (df64*)take((size_t)R * (NB / 8) * 8);
  s.v = (df64*)take((size_t)R * 8);
  s.tp = (float2*)take((size_t)R * (NB / 8) * 8);
  s.t = (float*)take((size_t)R * 4);
  s.e = (float*)take((size_t)R * 4);
  s.cw = (float*)take((size_t)M * 4);
  s.rexp = (int*)take((size_t)R * 4);
  s.mgen = (int*)take((size_t)R * 4);
  s.c = (int*)take((size_t)(M + 1) * 4);
  s.r = (int*)take((size_t)M * 4);
  if (out) *out = s;
  return o;
}
constexpr int DM_BAD = 1 << 20;   // exponent of a row or column with a non-finite entry
constexpr int DM_LOW = -400;      // the smallest exponent of a scaled row (2^-126 of a row and 2^-254 of a balance)
constexpr float DM_TRUST = 1024.f;   // a sixteenth of the scales, in the first digits' units (2^-7 of each scale)
constexpr int DM_MAX = 255;       // largest M: four pairs a lane, sums below 2^61

// Bk of one row (optional) and the sum k . Bk in double-float, by a warp: four columns a lane, B's entries of eight
// rows in flight together and split without a branch where all are ordinary numbers (entry by entry, one row in a
// thousand made N = 1000, M = 100, two outputs 122 us instead of 22; so, 50)
static __device__ __noinline__ df64 dm_row_general(const double* B, int b_pairs, const df64* k, const int* c, int M,
                                                   double* Bk) {
  constexpr int G = 8;
  const int lane = threadIdx.x & 31;
  df64 v = make_df(0.f);
  for (int b0 = lane; b0 - lane < M; b0 += 128) {
    df64 x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = make_df(0.f);
#pragma unroll 1
    for (int a0 = 0; a0 < M; a0 += G) {
      double e[G][4];
      bool plain = true;
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) e[g][j] = a0 + g < M && b0 + 32 * j < M ? B[(size_t)(a0 + g) * M + b0 + 32 * j] : 0.0;
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) plain = plain && df_plain(e[g][j]);
      auto group = [&](auto split) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const df64 ka = k[min(a0 + g, M - 1)];
#pragma unroll
          for (int j = 0; j < 4; ++j) acc_fma(x[j], split(e[g][j]), ka);
        }
      };
      if (b_pairs) group([](double w) { return make_df(__int_as_float(__double2loint(w)), __int_as_float(__double2hiint(w))); });
      else if (__all_sync(~0u, plain)) group([](double w) { return df_from_double_plain(w); });
      else group([](double w) { return df_from_double(w); });
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = acc_done(x[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = b0 + 32 * j;
      if (b < M) {
        if (c[b] >= DM_BAD) x[j] = make_df(__int_as_float(0x7fffffff));
        if (Bk) Bk[b] = df_to_double_int(x[j]);
        v = fma_(k[b], x[j], v);
      }
    }
  }
  return warp_sum(v);
}

__global__ void __launch_bounds__(DM_T, 1) det_mma_kernel(int N, int M, int Dout, const double* lsf2, const double* A,
                                                          const double* B, int b_pairs, const double* kin, double* Bk,
                                                          double* m_out, double* v_out, int NB, int nrt) {
  extern __shared__ __align__(16) char smem_raw[];
  const int R = 16 * nrt, KS = (M + 15) >> 4, NT = NB >> 3, MP = M | 1;
  DmSmem s;
  dm_carve(&s, smem_raw, M, NB, R);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = blockIdx.y;
  const int nblk = (M + NB) / NB;   // blocks of the M + 1 columns
  A += (size_t)d * M;
  B += (size_t)d * M * M;
  const float qnan = __int_as_float(0x7fffffff);
  __shared__ df64 s_sf2;
  const double lsf = lsf2[0];
  for (int i = tid; i < M; i += DM_T) s.c[i] = -126;
  // ---- the exponents of B's columns, then of its rows beside them.  A warp takes a row's columns by 128, four
  // such items' loads in flight; the entries' exponents wait in bytes (in the place of B's digits) for the second pass
  // |entry| < 2^ex_of: of a pair by its high word, of a float64 rounded as that word is (a NaN of all ones carries
  // out of the field, which stays above every exponent)
  auto ex_of = [&](double v, bool pair) {
    const int h = (int)(((unsigned)__double2loint(v) >> 23) & 0xffu);
    const int e = (int)((((unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL) + (1ULL << 28)) >> 52);
    return pair ? h - 126 : e - 1022;
  };
  const int EP = (M + 3) & ~3, hs = M > 128;   // bytes of a row; a row is 2^hs items
  unsigned char* const eb = reinterpret_cast<unsigned char*>(s.B);
  int ea[8];   // A's exponents
#pragma unroll
  for (int j = 0; j < 8; ++j) ea[j] = lane + 32 * j < M ? ex_of(A[lane + 32 * j], false) : 2 * DM_LOW;
  {
    const int cb = (warp & hs) * 128 + lane;   // (a warp's items are all of one side)
    int cm[4] = {-126, -126, -126, -126};
    for (int it = warp; it < M << hs; it += 4 * DM_W) {
      double v[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int a = (it + u * DM_W) >> hs;
          v[u][j] = a < M && cb + 32 * j < M ? B[(size_t)a * M + cb + 32 * j] : 0.0;
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int a = (it + u * DM_W) >> hs;
          const int e = min(max(ex_of(v[u][j], b_pairs), -126), 129);   // -126: zero or below the float range
          cm[j] = max(cm[j], e);
          if (a < M && cb + 32 * j < EP) eb[a * EP + cb + 32 * j] = (unsigned char)(e + 126);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (cb + 32 * j < M) atomicMax(&s.c[cb + 32 * j], cm[j] > 128 ? DM_BAD : cm[j]);
  }
  __syncthreads();
  {
    int cc[2][4], cmax = 0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = 4 * (lane + 32 * j) + u;
        cc[j][u] = c < M ? s.c[c] + 126 : DM_BAD;   // (a column with a NaN takes no part)
        if (cc[j][u] < DM_BAD) cmax = max(cmax, cc[j][u]);
      }
    for (int a = warp; a < M; a += DM_W) {
      int e = DM_LOW;
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (4 * (lane + 32 * j) < M) {
          const unsigned w = *reinterpret_cast<const unsigned*>(eb + a * EP + 4 * (lane + 32 * j));
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int b = (w >> (8 * u)) & 0xffu;
            if (b) e = max(e, b - cc[j][u]);
          }
        }
      e = __reduce_max_sync(~0u, e);
      if (lane == 0) s.r[a] = min(e, 0);
    }
    cmax = __reduce_max_sync(~0u, cmax) - 126;
    for (int i = tid; i < M; i += DM_T) {
      const int e = s.c[i] - cmax;
      s.cw[i] = e > 0 || e < -126 ? 0.f : pow2f(e);
    }
  }
  __syncthreads();
  {
    int e = 2 * DM_LOW;   // A's column, beside the rows' exponents (every warp alike)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (lane + 32 * j < M) e = max(e, ea[j] > 128 ? DM_BAD : ea[j] - s.r[lane + 32 * j]);
    e = __reduce_max_sync(~0u, e);
    if (lane == 0) s.c[M] = e;
    __syncwarp();
  }
  // ---- columns [c0, c0 + NB) of B' as digits; a lane's four entries of a column are the matrix
  // instruction's fragment, the next item's in flight while one is worked on
  auto stage_B = [&](int c0) {
    double r[4], rn[4];
    auto fetch = [&](int nt, int ks) {
      const int c = c0 + nt * 8 + (lane >> 2), a0 = ks * 16 + 2 * (lane & 3);
      const double* p = c == M ? A + a0 : B + (size_t)a0 * M + c;
      const size_t st = c == M ? 1 : M;
      const bool on = nt < NT && c <= M;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int o = (i & 1) + 8 * (i >> 1);
        rn[i] = on && a0 + o < M ? p[o * st] : 0.0;
      }
    };
    // fragment (column tile, k step) number warp, then every DM_W-th
    auto next = [&](int& nt, int& ks) {
      ks += DM_W;
      while (ks >= KS) ks -= KS, ++nt;
    };
    int nt0 = 0, ks0 = warp - DM_W;
    next(nt0, ks0);
    fetch(nt0, ks0);
    for (int nt = nt0, ks = ks0; nt < NT;) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = rn[i];
      const int c = c0 + nt * 8 + (lane >> 2), a0 = ks * 16 + 2 * (lane & 3), F = 52 - (c <= M ? s.c[c] : 0);
      uint2* q = reinterpret_cast<uint2*>(s.B) + (nt * KS + ks) * 32 + lane;
      next(nt, ks);
      if (nt < NT) fetch(nt, ks);
      const bool pair = b_pairs && c < M;
      long long t[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {   // (an exponent of DM_BAD gives zeros)
        const int a = a0 + (i & 1) + 8 * (i >> 1), Fa = F - (a < M ? s.r[a] : 0);
        df64 v = df_from_double(r[i]);   // (pairs and float64 give the same results)
        if (pair) v = make_df(__int_as_float(__double2loint(r[i])), __int_as_float(__double2hiint(r[i])));
        t[i] = fx_bits_by(v.hi, Fa) + fx_bits_by(v.lo, Fa);
      }
      unsigned w0[DM_S], w1[DM_S];
      digit_pairs(t[0], t[1], w0);
      digit_pairs(t[2], t[3], w1);
#pragma unroll
      for (int j = 0; j < DM_S; ++j) q[j * NT * KS * 32] = make_uint2(w0[j], w1[j]);
    }
  };
  if (nblk == 1) stage_B(0);
  if (tid == DM_T - 1) s_sf2 = df_from_double(exp(lsf));   // (read after the barriers of the first rows)
  const int ntile = (N + R - 1) / R;
  for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int n0 = tile * R, nr = min(R, N - n0);
    // ---- a warp a row: its largest exponent (|k'| < 2^ex), the integers k' 2^(-1 - ex) in units of 2^-53
    // and their digits (rows past nr keep stale digits: their results are not used)
    for (int r = warp; r < nr; r += DM_W) {
      const double* kr = kin + (size_t)(n0 + r) * M;
      double kv[4][2];
      int ex = DM_LOW;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int a = 2 * lane + 64 * i;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          kv[i][u] = a + u < M ? kr[a + u] : 0.0;
          ex = max(ex, (int)((__double_as_longlong(kv[i][u]) >> 52) & 0x7ff) - 1022 + (a + u < M ? s.r[a + u] : 0));
        }
      }
      ex = __reduce_max_sync(~0u, ex);
      if (ex > 128) ex = DM_BAD;
      unsigned* q0 = s.A + ((size_t)((r >> 4) * KS) * 32 + (r & 7) * 4) * 4 + ((r >> 3) & 1);
      float e = 0.f;
      bool full = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int p = lane + 32 * i;
        if (p < KS * 8) {
          long long t[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int a = 2 * p + u;
            t[u] = 0;
            if (a < M) {
              const df64 k = df_from_double(kv[i][u]);
              t[u] = digits_of(kv[i][u], ex - s.r[a]);
              s.k[r * MP + a] = k;
              full |= k.hi != 0.f;
              e = __fmaf_rn(fabsf(k.hi), s.cw[a], e);
            }
          }
          unsigned w[DM_S];
          digit_pairs(t[0], t[1], w);
          unsigned* q = q0 + ((p >> 3) * 32 + (p & 3)) * 4 + 2 * ((p >> 2) & 1);
#pragma unroll
          for (int j = 0; j < DM_S; ++j) q[(size_t)j * nrt * KS * 128] = w[j];
        }
      }
      e = warp_sum(e);
      full = __any_sync(~0u, full);
      if (lane == 0) {
        s.rexp[r] = ex;
        s.e[r] = full ? e : -1.f;
      }
    }
    for (int c0 = 0; c0 <= M; c0 += NB) {
      if (nblk > 1) stage_B(c0);
      __syncthreads();
      for (int it = warp; it < NT * nrt; it += DM_W) {
        const int rt = it / NT, nt = it - rt * NT;
        const uint4* fa = reinterpret_cast<const uint4*>(s.A) + (size_t)rt * KS * 32 + lane;
        const uint2* fb = reinterpret_cast<const uint2*>(s.B) + (size_t)nt * KS * 32 + lane;
        long long Z[4] = {0, 0, 0, 0};
        float mag[4] = {0.f, 0.f, 0.f, 0.f};   // (at most 255 2^14: exact)
        for (int k0 = 0; k0 < KS; k0 += 8) {
          float acc[DM_ACC][4];
#pragma unroll
          for (int i = 0; i < DM_ACC; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
          const int k1 = min(k0 + 8, KS);
#pragma unroll 2
          for (int ks = k0; ks < k1; ++ks)
            dm_step<false>(acc, mag, fa + ks * 32, nrt * KS * 32, fb + ks * 32, NT * KS * 32);
#pragma unroll
          for (int j = 0; j < 4; ++j) Z[j] += dm_fold(acc, j);
        }
        df64 v[2] = {make_df(0.f), make_df(0.f)};
        float t[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = rt * 16 + (lane >> 2) + 8 * (j >> 1), cl = nt * 8 + 2 * (lane & 3) + (j & 1), c = c0 + cl;
          if (r < nr && c <= M) {
            const int re = s.rexp[r], be = s.c[c];
            const df64 X = re >= DM_BAD || be >= DM_BAD ? make_df(qnan)
                                                       : scale2(df_of_int(Z[j], 58), max(-252, min(re + be + 6, 252)));
            if (c < M) {
              const df64 k = s.k[r * MP + c];
              if (Bk) Bk[((size_t)(n0 + r) * Dout + d) * M + c] = df_to_double_int(X);
              v[j >> 1] = fma_(k, X, v[j >> 1]);
              t[j >> 1] = __fmaf_rn(fabsf(k.hi) * s.cw[c], mag[j], t[j >> 1]);
            } else {
              s.mgen[r] = mag[j] < DM_TRUST && re < DM_BAD;
              if (m_out) m_out[(size_t)(n0 + r) * Dout + d] = df_to_double_int(X);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
          for (int o = 1; o < 4; o <<= 1) v[i] = add(v[i], shfl_xor(v[i], o));
          t[i] += __shfl_xor_sync(~0u, t[i], 1);
          const int o = (rt * 16 + (lane >> 2) + 8 * i) * NT + nt;
          if ((lane & 1) == 0) reinterpret_cast<float*>(s.tp + o)[(lane >> 1) & 1] = t[i];
          if ((lane & 3) == 0) s.vp[o] = v[i];
        }
      }
      __syncthreads();
      // ---- v: a warp a row, the column tiles' parts by one butterfly (NT <= 32)
      for (int r = warp; r < nr; r += DM_W) {
        df64 v = lane < NT ? s.vp[r * NT + lane] : make_df(0.f);
        const float2 t2 = lane < NT ? s.tp[r * NT + lane] : make_float2(0.f, 0.f);
        float t = t2.x + t2.y;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          v = add(v, shfl_xor(v, o));
          t += __shfl_xor_sync(~0u, t, o);
        }
        if (c0 > 0) {
          v = add(s.v[r], v);
          t += s.t[r];
        }
        if (c0 + NB <= M) {
          __syncwarp();
          if (lane == 0) {
            s.v[r] = v;
            s.t[r] = t;
          }
        } else {
          const float e = s.e[r];
          const size_t o = (size_t)(n0 + r) * Dout + d;
          if (s.rexp[r] < DM_BAD && e >= 0.f && !(e > 0.f && t >= DM_TRUST * e))
            v = dm_row_general(B, b_pairs, s.k + r * MP, s.c, M, Bk ? Bk + o * M : nullptr);
          if (s.mgen[r] && e >= 0.f && m_out && s.c[M] < DM_BAD) {
            df64 m = make_df(0.f);
            for (int a = lane; a < M; a += 32) m = fma_(s.k[r * MP + a], df_from_double(A[a]), m);
            m = warp_sum(m);
            if (lane == 0) m_out[o] = df_to_double_int(m);
          }
          if (lane == 0 && v_out) v_out[o] = df_to_double(add(s_sf2, v));
        }
      }
    }
  }
}

// elements of one det_bwd row buffer: RG rows of kfu (or dkfu) and Bk, x, dm, dv
__host__ __device__ inline int det_bwd_rowbuf(int RG, int M, int D, int Dk) { return RG * (M * (1 + Dk) + D + 2 * Dk); }

// Deterministic-input layer backward, per row (geepee/aep_models.py:451-460 with
// kfucompDer, kernels.py:381-399):
//   dkfu_nb = sum_d dm_nd A_db + 2 sum_d dv_nd Bk_ndb,   L_nb = dkfu_nb kfu_nb
//   dsf2 += sum L / sf2;  dl_q += sum L (x-z)^2 / l^{3/2};  dZ_bq += sum_n L (x_nq - z_bq)/l_q
//   dA_db += sum_n dm_nd kfu_nb;   dx_nq = -sum_b L_nb (x_nq - z_bq)/l_q   (optional)
// Threads are (b, row group): threadIdx.x is the pseudo-input b, threadIdx.y one of RG row
// groups; a CTA takes a contiguous range of rows, RG at a time, whose kfu, Bk, x, dm, dv rows
// are copied into shared memory (double-buffered: the next RG rows' copies are in flight while
// these compute) and converted once; Z and A likewise at the start.  Per-b sums (dZ, dA) are
// reduced over the row groups in shared memory and flushed with one write (or atomic) per CTA;
// dsf2 and dl by one CTA reduction.
// DB outputs (Dout <= DB, every one of the first DB live unless DB = DO_MAX) and EX (D == DC)
// are compile-time, so that the per-row loops carry no branch between independent sums.
template <typename T, int DC, int DB, bool EX>
__global__ void __launch_bounds__(512) det_bwd_kernel(int N, int M, int D, int Dout,
                                                      const typename Num<T>::store_t* x, int ldx,
                                                      const typename Num<T>::store_t* z, const double* lls2,
                                                      const double* lsf2, const typename Num<T>::store_t* A,
                                                      const typename Num<T>::store_t* kfu,
                                                      const typename Num<T>::store_t* Bk,
                                                      const typename Num<T>::store_t* dm,
                                                      const typename Num<T>::store_t* dv,
                                                      const typename Num<T>::store_t* dkfu, double* dsf2,
                                                      double* dl, double* dZ, double* dA,
                                                      typename Num<T>::store_t* dx, double* part,
                                                      long part_stride) {
  typedef typename Num<T>::store_t S;
  extern __shared__ __align__(16) char smem_raw[];
  float2* tab = reinterpret_cast<float2*>(smem_raw);
  Hyp<T>* h = reinterpret_cast<Hyp<T>*>(smem_raw + 256 * sizeof(float2));
  const int RG = blockDim.y, XW = blockDim.x >> 5;
  const int Dk = dkfu ? 0 : Dout;   // outputs whose A, Bk, dm, dv are read
  const int BS = det_bwd_rowbuf(RG, M, D, Dk);
  T* zs = reinterpret_cast<T*>(smem_raw + 256 * sizeof(float2) + sizeof(Hyp<T>));   // [M][D]
  T* as = zs + (size_t)M * D;                // [Dk][M]
  T* buf = as + (size_t)Dk * M;              // [2][BS]: RG rows of kfu (or dkfu), Bk, x, dm, dv
  T* red = buf + 2 * (size_t)BS;             // [RG][XW][DC] (dx) / [RG][blockDim.x][DC+DO_MAX]
  const int b = threadIdx.x, rg = threadIdx.y, lane = threadIdx.x & 31, xw = threadIdx.x >> 5;
  const int tid = rg * blockDim.x + b, nth = blockDim.x * blockDim.y;
  const int nbeg = (int)((long)N * blockIdx.x / gridDim.x), nend = (int)((long)N * (blockIdx.x + 1) / gridDim.x);
  // The rows of a pass arrive by asynchronous copies into one of two buffers while the other
  // pass computes; each thread converts the elements it copied (one conversion site for all
  // of them), and a barrier publishes them.  Buffer layout (nr <= RG rows from n0):
  //   [0, RG M) kfu or dkfu rows | [RG M, RG M (1+Dk)) Bk rows | RG D x rows | RG Dk dm | RG Dk dv
  auto rowbuf = [&](int i, int n0, int nr, bool convert) {
    T* B0 = buf + (size_t)(i & 1) * BS;
    S* R0 = reinterpret_cast<S*>(B0);
    const long nk = (long)nr * M, nb = (long)nr * Dk * M, nx = (long)nr * D, ng = (long)nr * Dk;
    const long ob = (long)RG * M, ox = ob + (long)RG * Dk * M, om = ox + (long)RG * D, ov = om + (long)RG * Dk;
    for (long e = tid; e < nk + nb + nx + 2 * ng; e += nth) {
      long o;
      const S* src;
      if (e < nk) {
        o = e;
        src = (dkfu ? dkfu : kfu) + (size_t)n0 * M + e;
      } else if (e < nk + nb) {
        o = ob + (e - nk);
        src = Bk + (size_t)n0 * Dk * M + (e - nk);
      } else if (e < nk + nb + nx) {
        const long t = e - nk - nb, r = t / D;
        o = ox + t;
        src = x + (size_t)(n0 + r) * ldx + (t - r * D);
      } else if (e < nk + nb + nx + ng) {
        o = om + (e - nk - nb - nx);
        src = dm + (size_t)n0 * Dk + (e - nk - nb - nx);
      } else {
        o = ov + (e - nk - nb - nx - ng);
        src = dv + (size_t)n0 * Dk + (e - nk - nb - nx - ng);
      }
      o = GPK_IDX(o, BS, 4);
      if (convert) {
        B0[o] = Num<T>::ld(R0[o]);
      } else {
        const unsigned d = (unsigned)__cvta_generic_to_shared(R0 + o);
        if (sizeof(S) == 8)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
        else
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src));
      }
    }
  };
  // Z and A the same way (with the first pass's rows)
  auto zabuf = [&](bool convert) {
    S* zr = reinterpret_cast<S*>(zs);
    for (long e = tid; e < (long)M * D + (long)Dk * M; e += nth) {
      const S* src = e < (long)M * D ? z + e : A + (e - (long)M * D);
      if (convert) {
        zs[e] = Num<T>::ld(zr[e]);
      } else {
        const unsigned d = (unsigned)__cvta_generic_to_shared(zr + e);
        if (sizeof(S) == 8)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
        else
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src));
      }
    }
  };
  zabuf(false);
  if (nbeg < nend) rowbuf(0, nbeg, min(RG, nend - nbeg), false);
  load_exp_table(tab);
  __syncthreads();
  load_hyp(*h, lls2, lsf2, D, tab);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  zabuf(true);
  if (nbeg < nend) rowbuf(0, nbeg, min(RG, nend - nbeg), true);
  __syncthreads();
  T zb[DC], gz[DC], gl[DC];
#pragma unroll
  for (int q = 0; q < DC; ++q) {
    zb[q] = (b < M && q < D) ? zs[b * D + q] : Num<T>::zero();
    gz[q] = gl[q] = Num<T>::zero();
  }
  T ab[DO_MAX], ga[DO_MAX];
#pragma unroll
  for (int d = 0; d < DO_MAX; ++d) {
    ab[d] = (b < M && d < Dk) ? as[d * M + b] : Num<T>::zero();
    ga[d] = Num<T>::zero();
  }
  T gsf = Num<T>::zero();
  auto q_on = [&](int q) { return EX || q < D; };
  auto d_on = [&](int d) { return d < DB && (DB < DO_MAX || d < Dout); };
  for (int n0 = nbeg, it = 0; n0 < nend; n0 += RG, ++it) {
    const int n = n0 + rg;
    const bool row = n < nend;
    const int nr = min(RG, nend - n0);
    const bool more = n0 + RG < nend;
    if (more) rowbuf(it + 1, n0 + RG, min(RG, nend - n0 - RG), false);   // the next pass's rows
    const T* B0 = buf + (size_t)(it & 1) * BS;
    const T* kr = B0 + (size_t)rg * M;
    const T* bkr = B0 + (size_t)RG * M + (size_t)rg * Dk * M;
    const T* xs = B0 + (size_t)RG * M * (1 + Dk) + (size_t)rg * D;
    const T* dmr = B0 + (size_t)RG * (M * (1 + Dk) + D) + (size_t)rg * Dk;
    const T* dvr = dmr + (size_t)RG * Dk;
    T L = Num<T>::zero();
    if (row && b < M) {
      const T k = kr[b];
      T g = Num<T>::zero();
      if (dkfu) {
        g = k;   // the staged row holds dkfu here
      } else {
#pragma unroll
        for (int d = 0; d < DB; ++d) {
          if (d_on(d)) {
            const T dmd = dmr[d], dvd = dvr[d];
            g = fma_(dmd, ab[d], g);
            g = fma_(scale2(dvd, 1), bkr[(size_t)d * M + b], g);
            ga[d] = fma_(dmd, k, ga[d]);
          }
        }
      }
      const T kk = dkfu ? Num<T>::ld(kfu[(size_t)n * M + b]) : k;
      L = mul(g, kk);
      gsf = add(gsf, L);
#pragma unroll
      for (int q = 0; q < DC; ++q) {
        if (q_on(q)) {
          const T df = sub(xs[q], zb[q]);
          const T t = mul(L, df);
          gz[q] = fma_(t, h->inv_l2[q], gz[q]);
          gl[q] = fma_(t, df, gl[q]);
        }
      }
    }
    if (dx) {
      // dx_nq = -sum_b L (x_nq - z_bq) / l_q: warp sums over b (all q in one butterfly), then
      // over the group's warps
#pragma unroll
      for (int c0 = 0; c0 < DC; c0 += 8) {   // eight dimensions per butterfly (register budget)
        T t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int q = c0 + u;
          t[u] = (q_on(q) && row && b < M) ? mul(L, mul(sub(xs[q], zb[q]), h->inv_l2[q])) : Num<T>::zero();
        }
        warp_sum_many<8>(t);   // lane l now holds the warp total of dimension c0 + l / 4
        const int q = c0 + (lane >> 2);
        if ((lane & 3) == 0 && q < D) red[(rg * XW + xw) * DC + q] = t[0];
      }
      __syncthreads();
      if (row && b < D) {
        T sacc = Num<T>::zero();
        for (int w = 0; w < XW; ++w) sacc = add(sacc, red[(rg * XW + w) * DC + b]);
        dx[(size_t)n * D + b] = Num<T>::st(neg(sacc));
      }
    }
    (void)nr;
    if (more) {   // the next pass's rows: this thread's copies landed; convert them, publish
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      rowbuf(it + 1, n0 + RG, min(RG, nend - n0 - RG), true);
    }
    __syncthreads();
  }
  // per-b sums over the row groups -> one write per CTA and (b, q) / (d, b): into this CTA's
  // partial block ([dZ M*D | dA Dout*M | dsf2 | dl D], fixed-order path) or atomically
  double* const pblk = part ? part + (size_t)blockIdx.x * part_stride : nullptr;
  T* pb = red;   // [RG][blockDim.x][DC + DO_MAX]
  const int W = DC + DO_MAX;
#pragma unroll
  for (int q = 0; q < DC; ++q) pb[(rg * blockDim.x + b) * W + q] = gz[q];
#pragma unroll
  for (int d = 0; d < DO_MAX; ++d) pb[(rg * blockDim.x + b) * W + DC + d] = ga[d];
  __syncthreads();
  if (rg == 0 && b < M) {
#pragma unroll
    for (int q = 0; q < DC; ++q) {
      if (q < D) {
        T sacc = pb[b * W + q];
        for (int r = 1; r < RG; ++r) sacc = add(sacc, pb[(r * blockDim.x + b) * W + q]);
        if (pblk) pblk[(size_t)b * D + q] = (double)Num<T>::st(sacc);
        else atomicAdd(&dZ[(size_t)b * D + q], (double)Num<T>::st(sacc));
      }
    }
    const bool wantA = dA && !dkfu;
#pragma unroll
    for (int d = 0; d < DO_MAX; ++d) {
      if (d < (dkfu ? 0 : Dout)) {
        T sacc = pb[b * W + DC + d];
        for (int r = 1; r < RG; ++r) sacc = add(sacc, pb[(r * blockDim.x + b) * W + DC + d]);
        if (pblk) pblk[(size_t)M * D + (size_t)d * M + b] = wantA ? (double)Num<T>::st(sacc) : 0.0;
        else if (wantA) atomicAdd(&dA[(size_t)d * M + b], (double)Num<T>::st(sacc));
      }
    }
  }
  __syncthreads();
  // dsf2 and dl: CTA reduction (the 1 + D warp sums in one butterfly, then lane i of warp 0
  // adds value i over the warps in order)
  const int wid = tid >> 5, nw = nth >> 5, ln = tid & 31;
  T* rw = red;   // [nw][1 + DC]
#pragma unroll
  for (int c0 = 0; c0 < 1 + DC; c0 += 8) {   // values 0 (sf2) and 1 + q (dimension q), eight at a time
    T vals[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = c0 + u;
      vals[u] = i == 0 ? gsf : (i <= DC ? gl[(i - 1) & (DC - 1)] : Num<T>::zero());
    }
    warp_sum_many<8>(vals);
    const int i = c0 + (ln >> 2);
    if ((ln & 3) == 0 && i < 1 + DC) rw[wid * (1 + DC) + i] = vals[0];
  }
  __syncthreads();
  if (wid == 0 && ln < 1 + DC) {
    T tot = rw[ln];
    for (int w = 1; w < nw; ++w) tot = add(tot, rw[w * (1 + DC) + ln]);
    const size_t o = (size_t)M * D + (size_t)(dkfu ? 0 : Dout) * M;
    if (ln == 0) {
      const double vsf = (double)Num<T>::st(div(tot, h->sf2));
      if (pblk) pblk[o] = vsf;
      else atomicAdd(dsf2, vsf);
    } else if (ln - 1 < D) {
      // d/d ell of exp(-(x-z)^2/(2 ell^2)) = (x-z)^2 / ell^3 = (x-z)^2 * (1/l)^{3/2}
      const int q = ln - 1;
      const T il = h->inv_l2[q];
      const double vl = (double)Num<T>::st(mul(tot, mul(il, sqrt_(il))));
      if (pblk) pblk[o + 1 + q] = vl;
      else atomicAdd(&dl[q], vl);
    }
  }
}

// Weighted Gram reduction:  C[d] += sum_n w[n,d] u_n v_n^T  (u, v: [N,M] rows; C: [Dout,M,M] f64)
// 32x32 output tile per CTA, n split across gridDim.z.  Rows are staged GB at a time, with
// all of a stage's global loads in flight together.  (The dBhat / dSucav einsums of
// geepee/aep_models.py:463-464, 490-493.)
constexpr int GB = 32;
template <typename T>
__global__ void __launch_bounds__(256) gram_kernel(int N, int M, int Dout, const typename Num<T>::store_t* u,
                                                   const typename Num<T>::store_t* v,
                                                   const typename Num<T>::store_t* w, double* C, int sym,
                                                   double* part) {
  typedef typename Num<T>::store_t S;
  __shared__ T su[GB][32], sv[GB][32], sw[GB][DO_MAX];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 8 rows of threads, 4 outputs each
  // sym (u == v, C symmetric): blockIdx.x enumerates the tiles bi <= bj only, and an
  // off-diagonal tile is added at both (i, j) and (j, i)
  int bi = blockIdx.y, bj = blockIdx.x;
  if (sym) {
    const int nt = (M + 31) >> 5;
    bi = 0;
    bj = blockIdx.x;
    while (bj >= nt - bi) {
      bj -= nt - bi;
      ++bi;
    }
    bj += bi;
  }
  const int i0 = bi * 32, j0 = bj * 32;
  T acc[DO_MAX][4];
#pragma unroll
  for (int d = 0; d < DO_MAX; ++d)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[d][r] = Num<T>::zero();
  const int nbeg = (int)((long)N * blockIdx.z / gridDim.z), nend = (int)((long)N * (blockIdx.z + 1) / gridDim.z);
  for (int n0 = nbeg; n0 < nend; n0 += GB) {
    // stage rows n0 .. n0+GB-1: element e = tid + 256 p of the u and v tiles (row e/32, col e%32)
    S ru[4], rv[4], rw = S(0);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int e = threadIdx.x + 256 * p, rl = e >> 5, c = e & 31, n = n0 + rl;
      ru[p] = (n < nend && i0 + c < M) ? u[(size_t)n * M + i0 + c] : S(0);
      rv[p] = (n < nend && j0 + c < M) ? v[(size_t)n * M + j0 + c] : S(0);
    }
    {
      const int rl = threadIdx.x / DO_MAX, d = threadIdx.x % DO_MAX, n = n0 + rl;
      if (rl < GB && d < Dout && n < nend) rw = w[(size_t)n * Dout + d];
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int e = threadIdx.x + 256 * p;
      su[e >> 5][e & 31] = Num<T>::ld(ru[p]);
      sv[e >> 5][e & 31] = Num<T>::ld(rv[p]);
    }
    if (threadIdx.x < GB * DO_MAX) sw[threadIdx.x / DO_MAX][threadIdx.x % DO_MAX] = Num<T>::ld(rw);
    __syncthreads();
    const int nr = min(GB, nend - n0);
    for (int rl = 0; rl < nr; ++rl) {
      const T vj = sv[rl][tx];
#pragma unroll
      for (int d = 0; d < DO_MAX; ++d) {
        if (d < Dout) {
          const T wv = mul(sw[rl][d], vj);
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[d][r] = fma_(su[rl][ty * 4 + r], wv, acc[d][r]);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int d = 0; d < DO_MAX; ++d) {
    if (d < Dout) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        int i = i0 + ty * 4 + r, j = j0 + tx;
        if (i < M && j < M) {
          const double val = (double)Num<T>::st(acc[d][r]);
          if (part) {   // fixed-order path: this row chunk's partial matrices, plain stores
            double* pc = part + (size_t)blockIdx.z * Dout * M * M;
            pc[((size_t)d * M + i) * M + j] = val;
            if (sym && bi != bj) pc[((size_t)d * M + j) * M + i] = val;
          } else {
            atomicAdd(&C[((size_t)d * M + i) * M + j], val);
            if (sym && bi != bj) atomicAdd(&C[((size_t)d * M + j) * M + i], val);
          }
        }
      }
    }
  }
}

// Symmetric weighted Gram reduction by unordered pairs:  C[d] += sum_n w[n,d] u_n u_n^T
// (the dBhat einsum of geepee/aep_models.py:463-464 with u = kfu).  A CTA owns GP_PPT pairs
// (a >= b, row-major lower-triangle order) per thread of one pair block and one chunk of rows
// (blockIdx.y); the chunk's rows go through shared memory GR at a time, and each pair's sum
// over the chunk is one product u_a u_b per row and one multiply-add per output.  Every pair is
// computed once (no tile padding, no lower half of diagonal tiles); the chunk's sums leave as a
// partial block of packed pairs for the fixed-order reduction.
constexpr int GP_PPT = 2;
constexpr int GP_T = 512;
template <typename T, int DB>
__global__ void __launch_bounds__(GP_T) gram_pairs_kernel(int N, int M, int Dout, const typename Num<T>::store_t* u,
                                                          const typename Num<T>::store_t* w, double* part,
                                                          long pstride, int GR) {
  typedef typename Num<T>::store_t S;
  extern __shared__ __align__(16) char smem_raw[];
  T* us = reinterpret_cast<T*>(smem_raw);   // [GR][M]
  T* ws = us + (size_t)GR * M;              // [GR][DO_MAX]
  const int tid = threadIdx.x, P = M * (M + 1) / 2;
  int ia[GP_PPT], ib[GP_PPT], pp[GP_PPT];
#pragma unroll
  for (int k = 0; k < GP_PPT; ++k) {
    pp[k] = blockIdx.x * (GP_T * GP_PPT) + tid + GP_T * k;
    tri_pair(pp[k] < P ? pp[k] : 0, ia[k], ib[k]);   // pairs past P compute (0, 0), never stored
  }
  // DB (compile-time) outputs per pair, so that the loop below has no branch between the
  // independent sums (DB = 4 serves Dout = 3 with a zero weight)
  T acc[GP_PPT][DB];
#pragma unroll
  for (int k = 0; k < GP_PPT; ++k)
#pragma unroll
    for (int d = 0; d < DB; ++d) acc[k][d] = Num<T>::zero();
  const int nbeg = (int)((long)N * blockIdx.y / gridDim.y), nend = (int)((long)N * (blockIdx.y + 1) / gridDim.y);
  for (int n0 = nbeg; n0 < nend; n0 += GR) {
    const int nr = min(GR, nend - n0);
    stage_async(reinterpret_cast<S*>(us), u + (size_t)n0 * M, (long)nr * M, tid, GP_T);
    for (int e = tid; e < nr * DO_MAX; e += GP_T) {
      const int r = e / DO_MAX, d = e - r * DO_MAX;
      ws[e] = d < Dout ? Num<T>::ld(w[(size_t)(n0 + r) * Dout + d]) : Num<T>::zero();
    }
    __syncthreads();
    convert_in_place(us, (long)nr * M, tid, GP_T);
    __syncthreads();
    for (int rl = 0; rl < nr; ++rl) {
      const T* ur = us + (size_t)rl * M;
      T wd[DB];
#pragma unroll
      for (int d = 0; d < DB; ++d) wd[d] = ws[rl * DO_MAX + d];
#pragma unroll
      for (int k = 0; k < GP_PPT; ++k) {
        const T kk = mul(ur[ia[k]], ur[ib[k]]);
#pragma unroll
        for (int d = 0; d < DB; ++d) acc[k][d] = fma_(wd[d], kk, acc[k][d]);
      }
    }
    __syncthreads();   // the rows are consumed before the next chunk overwrites them
  }
  double* pb = part + (size_t)blockIdx.y * pstride;
#pragma unroll
  for (int k = 0; k < GP_PPT; ++k) {
    if (pp[k] < P) {
#pragma unroll
      for (int d = 0; d < DB; ++d)
        if (d < Dout) pb[(size_t)d * P + pp[k]] = (double)Num<T>::st(acc[k][d]);
    }
  }
}

// ---- the symmetric weighted Gram reduction on the tensor cores (float64) ----
// C[d]_ab = sum_n (w u_a 2^-h)(u_b 2^h) over a chunk of rows for one output d, by the digit products of
// det_mma_kernel: the contraction runs over n, so each column of either factor is scaled by its largest entry
// of the rows staged (at most 128, so that the digit sums stay exact), and the staged sums, exact
// integers, are added up in float64.  h is half of w's exponent: both factors are then sqrt|w| u in size,
// and the staged sum is off by some 2^-52 of max_n sqrt|w| |u_a| max_n sqrt|w| |u_b| a row, however w and u grow
// along n.  Where the sum of |terms|, estimated from the first digits, is below 1/32 of that product (two columns
// that hardly meet), the staged rows are summed in double-float instead: every C_ab is good to some n 2^-47 of its
// own sum of |terms|, as a double-float sum is.  A CTA of 12 warps owns up to 60 of the 16 x 8 tiles on and below the
// diagonal, five a warp, their float64 sums in registers; the next rows arrive by asynchronous copies while
// these are multiplied.  The chunk's sums leave as a partial block of packed pairs for the
// fixed-order reduction.
// N = 20000, M = 100, two outputs, with the reduction 99 us (361 in double-float pairs), a third of it in the matrix
// pipe, the rest in digits and folds (87 with h = 0 and every result trusted); N = 1000 22 us (30).  Two
// input dimensions (2% of the results weak) 132 us, one with a lengthscale of 0.04 of the range (most of them) 359.
constexpr long GM_PAIRS = 1L << 20;
constexpr float GM_TRUST = 512.f;   // 1/32 of the scales, in the first digits' units
constexpr int GM_T = 384, GM_W = GM_T / 32, GM_TW = 5;
struct GmSmem {
  unsigned *A, *B;   // digits of w u and of u, as in DmSmem (the columns in the place of the rows)
  double *raw, *w;   // [16 KS][M], [16 KS]
  int *h, *aexp, *bexp;   // [16 KS] half of w's exponent; [M] of the columns of the two factors
  int* list;         // [GM_W][32] a warp's weak results: first time << 31 | row << 16 | column
};
__host__ __device__ inline size_t gm_carve(GmSmem* out, char* base, int M, int KS) {
  GmSmem s;
  size_t o = 0;
  auto take = [&](size_t n) {
    char* p = base + o;
    o += (n + 15) & ~(size_t)15;
    return p;
  };
  const int RT = (M + 15) >> 4, CT = (M + 7) >> 3;
  s.A = (unsigned*)take((size_t)DM_S * RT * KS * 512);
  s.B = (unsigned*)take((size_t)DM_S * CT * KS * 256);
  s.raw = (double*)take((size_t)16 * KS * M * 8);
  s.w = (double*)take((size_t)16 * KS * 8);
  s.h = (int*)take((size_t)16 * KS * 4);
  s.aexp = (int*)take((size_t)M * 4);
  s.bexp = (int*)take((size_t)M * 4);
  s.list = (int*)take((size_t)GM_W * 32 * 4);
  if (out) *out = s;
  return o;
}
// tiles on and below the diagonal: row i of 16 has min(2 i + 2, CT) of 8 columns
__host__ __device__ inline int gm_tiles(int M) {
  const int RT = (M + 15) >> 4, CT = (M + 7) >> 3;
  return RT * (RT - 1) + (CT < 2 * RT ? CT : 2 * RT);
}
__global__ void __launch_bounds__(GM_T, 1) gram_mma_kernel(int N, int M, int Dout, const double* u, const double* w,
                                                           double* part, long pstride, int rows, int KSM,
                                                           int tw) {
  extern __shared__ __align__(16) char smem_raw[];
  GmSmem s;
  gm_carve(&s, smem_raw, M, KSM);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = blockIdx.y;
  const int RT = (M + 15) >> 4, CT = (M + 7) >> 3, ntile = gm_tiles(M);
  const int nbeg = blockIdx.x * rows, nend = min(N, nbeg + rows);
  double C[GM_TW][4];
  int ti[GM_TW], tj[GM_TW];   // the warp's tiles (row -1: none)
#pragma unroll
  for (int i = 0; i < GM_TW; ++i) {
    int t = blockIdx.z * (GM_W * tw) + warp + GM_W * i, r = 0;
    const bool on = i < tw && t < ntile;
    if (!on) t = 0;
    while (t >= min(2 * r + 2, CT)) t -= min(2 * r + 2, CT), ++r;
    ti[i] = on ? r : -1;
    tj[i] = t;
#pragma unroll
    for (int j = 0; j < 4; ++j) C[i][j] = 0.0;
  }
  // the rows by steps of 16, as evenly as at most KSM steps at a time allow (few rows leave more results weak)
  const int steps = (nend - nbeg + 15) >> 4, nst = (steps + KSM - 1) / KSM;
  auto begin = [&](int st) { return min(nend, nbeg + 16 * (int)((long)steps * st / nst)); };
  auto fetch = [&](int st) {
    const int n0 = begin(st), nr = begin(st + 1) - n0;
    for (int e = tid; e < nr * M; e += GM_T) async_copy(s.raw + e, u + (size_t)n0 * M + e);
    for (int e = tid; e < nr; e += GM_T) async_copy(s.w + e, w + (size_t)(n0 + e) * Dout + d);
  };
  auto expo = [](double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7ff) - 1022; };   // |v| < 2^expo
  double* const pb = part + (size_t)blockIdx.x * pstride + (size_t)d * (M * (M + 1) / 2);
  unsigned seen = 0;   // results that were weak before: their sums stand in the partial block
  fetch(0);
  for (int st = 0; st < nst; ++st) {
    const int n0 = begin(st), nr = begin(st + 1) - n0, KS = (nr + 15) >> 4;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // ---- the columns' largest exponents (of w u at most: the factors' sum)
    for (int i = tid; i < M; i += GM_T) s.aexp[i] = s.bexp[i] = DM_LOW;
    for (int r = tid; r < nr; r += GM_T) s.h[r] = expo(s.w[r]) >> 1;
    __syncthreads();
    for (int c = tid & 127; c < M; c += 128) {
      int ea = DM_LOW, eb = DM_LOW;
      for (int r = tid >> 7; r < nr; r += GM_T / 128) {
        const int e = expo(s.raw[r * M + c]), f = expo(s.w[r]), h = s.h[r];
        eb = max(eb, e == 1025 ? DM_BAD : e + h);
        ea = max(ea, max(e, f) == 1025 ? DM_BAD : e + f - h);
      }
      atomicMax(&s.bexp[c], eb > 300 ? DM_BAD : eb);
      atomicMax(&s.aexp[c], ea > 300 ? DM_BAD : ea);
    }
    __syncthreads();
    // ---- digits: a lane's four rows of one column
    for (int f = warp; f < 2 * RT * KS; f += GM_W) {
      const int ks = f / (2 * RT), c8 = f - ks * 2 * RT, c = c8 * 8 + (lane >> 2), r0 = ks * 16 + 2 * (lane & 3);
      long long ta[4], tb[4];
      const int ea = c < M ? s.aexp[c] : 0, eb = c < M ? s.bexp[c] : 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + (i & 1) + 8 * (i >> 1);
        const bool on = c < M && r < nr;
        const double v = on ? s.raw[r * M + c] : 0.0, wv = on ? s.w[r] : 0.0;
        const int h = on ? s.h[r] : 0;
        ta[i] = digits_of(v * wv, ea + h);
        tb[i] = digits_of(v, eb - h);
      }
      unsigned w0[DM_S], w1[DM_S];
      digit_pairs(ta[0], ta[1], w0);
      digit_pairs(ta[2], ta[3], w1);
      unsigned* q = s.A + ((size_t)((c8 >> 1) * KSM + ks) * 32 + lane) * 4 + (c8 & 1);
#pragma unroll
      for (int j = 0; j < DM_S; ++j) {
        q[j * RT * KSM * 128] = w0[j];
        q[j * RT * KSM * 128 + 2] = w1[j];
      }
      if (c8 < CT) {
        digit_pairs(tb[0], tb[1], w0);
        digit_pairs(tb[2], tb[3], w1);
        uint2* p = reinterpret_cast<uint2*>(s.B) + (size_t)(c8 * KSM + ks) * 32 + lane;
#pragma unroll
        for (int j = 0; j < DM_S; ++j) p[j * CT * KSM * 32] = make_uint2(w0[j], w1[j]);
      }
    }
    __syncthreads();
    if (st + 1 < nst) fetch(st + 1);
    unsigned weak = 0;   // the results (bit 4 i + j: result j of tile i) that the digits are too coarse for
#pragma unroll
    for (int i = 0; i < GM_TW; ++i) {
      if (ti[i] < 0) continue;   // (uniform over the warp)
      float acc[DM_ACC][4], mag[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < DM_ACC; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[k][j] = 0.f;
      const uint4* fa = reinterpret_cast<const uint4*>(s.A) + (size_t)ti[i] * KSM * 32 + lane;
      const uint2* fb = reinterpret_cast<const uint2*>(s.B) + (size_t)tj[i] * KSM * 32 + lane;
#pragma unroll 1
      for (int ks = 0; ks < KS; ++ks) dm_step<true>(acc, mag, fa + ks * 32, RT * KSM * 32, fb + ks * 32, CT * KSM * 32);
      const bool strong = __all_sync(~0u, fminf(fminf(mag[0], mag[1]), fminf(mag[2], mag[3])) >= GM_TRUST);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int a = ti[i] * 16 + (lane >> 2) + 8 * (j >> 1), b = tj[i] * 8 + 2 * (lane & 3) + (j & 1);
        const int ea = a < M ? s.aexp[a] : 0, eb = b < M ? s.bexp[b] : 0, e = ea + eb;
        // 2^(e - 52), or NaN
        const double f = __hiloint2double(e >= DM_BAD / 2 ? 0x7fffffff : (e + 971) << 20, 0);
        if (!strong && mag[j] < GM_TRUST && a < M && b <= a && max(ea, eb) < DM_BAD && min(ea, eb) > DM_LOW)
          weak |= 1u << (4 * i + j);   // (not: a column of zeros)
        else
          C[i][j] = fma(__ll2double_rn(dm_fold(acc, j)), f, C[i][j]);
      }
    }
    if (__syncthreads_or(weak)) {
      // ---- the weak results: the staged rows once more, u and w u as double-floats in the place of the digits,
      // and each warp's results in turn, 32 at a time, a lane each (14 instructions a row)
      df64* const ud = reinterpret_cast<df64*>(s.B);
      df64* const wu = reinterpret_cast<df64*>(s.A);
      for (int r0 = warp; r0 < nr; r0 += 3 * GM_W) {   // a warp a row, three rows' loads in flight
        for (int c0 = lane; c0 < M; c0 += 128) {
          double v[3][4], wv[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int r = r0 + k * GM_W;
            wv[k] = r < nr ? w[(size_t)(n0 + r) * Dout + d] : 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[k][j] = r < nr && c0 + 32 * j < M ? u[(size_t)(n0 + r) * M + c0 + 32 * j] : 0.0;
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int r = r0 + k * GM_W;
            const df64 wd = df_from_double(wv[k]);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (r < nr && c0 + 32 * j < M) {
                const df64 x = df_from_double(v[k][j]);
                ud[r * M + c0 + 32 * j] = x;
                wu[r * M + c0 + 32 * j] = mul(wd, x);
              }
          }
        }
      }
      int first = __popc(weak);   // this lane's first in the warp's order
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(~0u, first, o);
        first += lane >= o ? x : 0;
      }
      const int total = __shfl_sync(~0u, first, 31);
      first -= __popc(weak);
      __syncthreads();
      int* const list = s.list + warp * 32;
      for (int t0 = 0; t0 < total; t0 += 32) {
        int k = first - t0;   // the place of this lane's next result among the 32
        if (k < 32 && k + __popc(weak) > 0) {
#pragma unroll
          for (int i = 0; i < GM_TW; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if ((weak >> (4 * i + j)) & 1u) {
                if (k >= 0 && k < 32)
                  list[k] = ((seen >> (4 * i + j)) & 1u ? 0 : (int)0x80000000) |
                            (ti[i] * 16 + (lane >> 2) + 8 * (j >> 1)) << 16 | (tj[i] * 8 + 2 * (lane & 3) + (j & 1));
                ++k;
              }
        }
        __syncwarp();
        if (t0 + lane < total) {
          const int c = list[lane], a = (c >> 16) & 0x7fff, b = c & 0xffff;
          const df64 *pa = wu + a, *pu = ud + b;
          df64 x = make_df(0.f);
#pragma unroll 4
          for (int r = 0; r < nr; ++r) {
            const df64 p = pa[r * M], q = pu[r * M];
            acc_fma(x, p, q);
          }
          double* const o = pb + a * (a + 1) / 2 + b;
          *o = df_to_double(acc_done(x)) + (c < 0 ? 0.0 : *o);
        }
        __syncwarp();
      }
      seen |= weak;
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < GM_TW; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = ti[i] * 16 + (lane >> 2) + 8 * (j >> 1), b = tj[i] * 8 + 2 * (lane & 3) + (j & 1);
      if (ti[i] >= 0 && a < M && b <= a) {
        double* const o = pb + a * (a + 1) / 2 + b;
        *o = (seen >> (4 * i + j)) & 1u ? *o + C[i][j] : C[i][j];
      }
    }
  }
}

// c[d] += sum_n w[n,d] u_n  (u: [N,M]; c: [Dout,M] f64).  32 columns per CTA, rows split over
// 8 warps and gridDim.y; each thread keeps WU rows' loads in flight at a time.
constexpr int WU = 4;
template <typename T>
__global__ void __launch_bounds__(256) wsum_kernel(int N, int M, int Dout, const typename Num<T>::store_t* u,
                                                   const typename Num<T>::store_t* w, double* c) {
  typedef typename Num<T>::store_t S;
  const int j = blockIdx.x * 32 + (threadIdx.x & 31);
  const int part = threadIdx.x >> 5;  // 8 n-partitions per CTA
  __shared__ T red[8][32][DO_MAX];
  T acc[DO_MAX];
#pragma unroll
  for (int d = 0; d < DO_MAX; ++d) acc[d] = Num<T>::zero();
  const int stride = gridDim.y * 8;
  if (j < M) {
    for (int n0 = blockIdx.y * 8 + part; n0 < N; n0 += stride * WU) {
      S ru[WU], rw[WU][DO_MAX];
#pragma unroll
      for (int t = 0; t < WU; ++t) {
        const int n = n0 + t * stride;
        ru[t] = n < N ? u[(size_t)n * M + j] : S(0);
#pragma unroll
        for (int d = 0; d < DO_MAX; ++d) rw[t][d] = (n < N && d < Dout) ? w[(size_t)n * Dout + d] : S(0);
      }
#pragma unroll
      for (int t = 0; t < WU; ++t) {
        const T uv = Num<T>::ld(ru[t]);
#pragma unroll
        for (int d = 0; d < DO_MAX; ++d)
          if (d < Dout) acc[d] = fma_(Num<T>::ld(rw[t][d]), uv, acc[d]);
      }
    }
  }
#pragma unroll
  for (int d = 0; d < DO_MAX; ++d) red[part][threadIdx.x & 31][d] = acc[d];
  __syncthreads();
  if (part == 0 && j < M) {
    for (int d = 0; d < Dout && d < DO_MAX; ++d) {
      T s = red[0][threadIdx.x][d];
      for (int p = 1; p < 8; ++p) s = add(s, red[p][threadIdx.x][d]);
      atomicAdd(&c[(size_t)d * M + j], (double)Num<T>::st(s));
    }
  }
}

// the tensor-core contraction, 1 <= M <= DM_MAX (8 columns and 16 rows always fit)
int dm_launch(int N, int M, int Dout, const double* lsf2, const double* A, const double* B, int b_pairs,
              const double* kin, double* Bk, double* m_out, double* v_out, cudaStream_t st) {
  const size_t cap = (size_t)227 * 1024 - 64;
  // as few column blocks as fit beside 16 rows (sizes only: the order of v's sum)
  int nblk = 1, NB = 0;
  for (;; ++nblk) {
    NB = 8 * gpk::ceil_div(gpk::ceil_div(M + 1, nblk), 8);
    if (dm_carve(nullptr, nullptr, M, NB, 16) <= cap) break;
  }
  // one CTA an SM over the outputs; 32 or 64 rows at a time once a CTA has that many
  const int gx = std::max(1, gpk::sm_count() / Dout), per = gpk::ceil_div(N, gx);
  int nrt = per <= 16 ? 1 : (per <= 32 ? 2 : 4);
  while (nrt > 1 && dm_carve(nullptr, nullptr, M, NB, 16 * nrt) > cap) nrt >>= 1;
  const size_t sm = dm_carve(nullptr, nullptr, M, NB, 16 * nrt);
  gpk::allow_smem(det_mma_kernel, sm, 64);
  det_mma_kernel<<<dim3(std::min(gx, gpk::ceil_div(N, 16 * nrt)), Dout), DM_T, sm, st>>>(
      N, M, Dout, lsf2, A, B, b_pairs, kin, Bk, m_out, v_out, NB, nrt);
  return gpk::check_launch("det_mma");
}

size_t det_fwd_smem(int M, int D, bool zstage, size_t tsz) {
  return 256 * 8 + sizeof(Hyp<df64>) + ((size_t)FT * M + FKA * FCB + 8 * DO_MAX * FT + FT * D + (zstage ? (size_t)M * D : 0)) * tsz;
}
size_t det_bwd_smem(int bx, int rg, int dc, int M, int D, int Dk, size_t tsz) {
  const size_t red = (size_t)rg * bx * (dc + DO_MAX);   // the largest of the three uses of the area
  return 256 * 8 + sizeof(Hyp<df64>) +
         ((size_t)M * D + (size_t)Dk * M + 2 * (size_t)det_bwd_rowbuf(rg, M, D, Dk) + red) * tsz;
}

int kern_fx_launch(int N, int M, int D, const double* x, int ldx, const double* z, int ldz, const double* lls2,
                   const double* lsf2, double* K, int ldk, cudaStream_t st) {
  // column blocks times as many row groups as keep the chip full in one wave
  const long nmb = gpk::ceil_div(M, FC), ntile = gpk::ceil_div(N, FR);
  const long rg = std::min(ntile, std::max(1L, (long)gpk::sm_count() * FCTA / nmb));
  const size_t sm = kFxTab * sizeof(float2) + sizeof(ArdHyp) + ((size_t)2 * FR * D + (size_t)FC * (D | 1)) * 16;
  gpk::allow_smem(kern_fx_kernel, sm);
  kern_fx_kernel<<<(unsigned)(nmb * rg), 256, sm, st>>>(N, M, D, x, ldx, z, ldz, lls2, lsf2, K, ldk);
  return gpk::check_launch("kern");
}

template <typename T>
int kern_launch(int N, int M, int D, const void* x, int ldx, const void* z, int ldz, const double* lls2,
                const double* lsf2, double jitter, void* K, int ldk, cudaStream_t st) {
  typedef typename Num<T>::store_t S;
  const dim3 grid(gpk::ceil_div(M, KC), gpk::ceil_div(N, KR));
  GPK_REQUIRE(grid.y <= 65535, "kern: N=%d too large (at most %d rows)", N, 65535 * KR);
  const size_t sm = 256 * sizeof(float2) + sizeof(Hyp<T>) + (size_t)(KR + KC) * D * sizeof(T);
  auto k = kern_matrix_kernel<T>;
  gpk::allow_smem(k, sm);
  k<<<grid, 256, sm, st>>>(N, M, D, (const S*)x, ldx, (const S*)z, ldz, lls2, lsf2, jitter, (S*)K, ldk);
  return gpk::check_launch("kern");
}

}  // namespace

extern "C" int gpk_kern(int prec, int N, int M, int D, const void* x, int ldx, const void* z, int ldz,
                        const double* lls2, const double* lsf2, double jitter, void* K, int ldk, void* stream) {
  GPK_NVTX("gpk_kern");
  GPK_REQUIRE(N >= 0 && M >= 0 && D >= 1 && D <= DMAXK, "kern: bad sizes N=%d M=%d D=%d", N, M, D);
  GPK_REQUIRE(x && z && lls2 && lsf2 && K, "kern: null pointer");
  GPK_REQUIRE(ldx >= D && ldz >= D && ldk >= M, "kern: bad leading dimension");
  if (N == 0 || M == 0) return GPK_OK;
  cudaStream_t st = gpk::as_stream(stream);
  // with a jitter the matrix goes into a factorisation, which amplifies its last bits by a condition
  // number of up to 1e7: it keeps the double-float evaluation (its M x M entries cost ~10 us)
  if (prec == GPK_DF64 && jitter != 0.0) return kern_launch<df64>(N, M, D, x, ldx, z, ldz, lls2, lsf2, jitter, K, ldk, st);
  // (one limit for every form, that of kern_matrix_kernel's grid)
  GPK_REQUIRE(gpk::ceil_div(N, KR) <= 65535, "kern: N=%d too large (at most %d rows)", N, 65535 * KR);
  if (prec == GPK_DF64)
    return kern_fx_launch(N, M, D, (const double*)x, ldx, (const double*)z, ldz, lls2, lsf2, (double*)K, ldk, st);
  if (prec == GPK_FP32) return kern_launch<float>(N, M, D, x, ldx, z, ldz, lls2, lsf2, jitter, K, ldk, st);
  return gpk::fail(GPK_EINVAL, "kern: unknown precision %d", prec);
}

extern "C" int gpk_det_fwd(int prec, int N, int M, int D, int Dout, const void* x, int ldx, const void* Z,
                           const double* lls2, const double* lsf2, const void* A, const void* B, void* kfu,
                           void* Bk, void* m_out, void* v_out, void* stream) {
  GPK_NVTX("gpk_det_fwd");
  GPK_REQUIRE(N >= 0 && M >= 1 && M <= 1024 && D >= 1 && D <= DMAXK, "det_fwd: bad sizes N=%d M=%d D=%d", N, M, D);
  GPK_REQUIRE(Dout >= 1 && Dout <= DO_MAX, "det_fwd: Dout=%d outside [1,%d]", Dout, DO_MAX);
  GPK_REQUIRE(x && Z && lls2 && lsf2 && A && B, "det_fwd: null input");
  if (N == 0) return GPK_OK;
  cudaStream_t st = gpk::as_stream(stream);
  // the kernel rows, then the contraction from them (where the caller takes the rows)
  if (prec == GPK_DF64 && kfu && M <= DM_MAX) {
    const int rc = kern_fx_launch(N, M, D, (const double*)x, ldx, (const double*)Z, D, lls2, lsf2, (double*)kfu, M, st);
    if (rc != GPK_OK) return rc;
    return dm_launch(N, M, Dout, lsf2, (const double*)A, (const double*)B, 0, (const double*)kfu, (double*)Bk,
                     (double*)m_out, (double*)v_out, st);
  }
  // one CTA column per output d; row tiles up to two resident CTAs per SM in all
  int gx = gpk::ceil_div(N, FT);
  const int cap = std::max(1, gpk::sm_count() * 2 / Dout);
  if (gx > cap) gx = cap;
  const dim3 grid(gx, Dout);
  const int zstage = (size_t)M * D * sizeof(df64) <= 32 * 1024;
  if (prec == GPK_DF64) {
    size_t sm = det_fwd_smem(M, D, zstage, sizeof(df64));
    auto k = det_fwd_kernel<df64>;
    gpk::allow_smem(k, sm);
    k<<<grid, 256, sm, st>>>(N, M, D, Dout, (const double*)x, ldx, (const double*)Z, lls2, lsf2,
                             (const double*)A, (const double*)B, (double*)kfu, (double*)Bk, (double*)m_out,
                             (double*)v_out, zstage);
  } else if (prec == GPK_FP32) {
    size_t sm = det_fwd_smem(M, D, zstage, sizeof(float));
    auto k = det_fwd_kernel<float>;
    gpk::allow_smem(k, sm);
    k<<<grid, 256, sm, st>>>(N, M, D, Dout, (const float*)x, ldx, (const float*)Z, lls2, lsf2, (const float*)A,
                             (const float*)B, (float*)kfu, (float*)Bk, (float*)m_out, (float*)v_out, zstage);
  } else {
    return gpk::fail(GPK_EINVAL, "det_fwd: unknown precision %d", prec);
  }
  return gpk::check_launch("det_fwd");
}

namespace {
template <typename T, int DB>
void contract_launch(int N, int M, int Dout, const void* kfu, const double* lsf2, const void* A, const void* B,
                     void* Bk, void* m_out, void* v_out, cudaStream_t st) {
  typedef typename Num<T>::store_t S;
  const size_t sm = det_contract_smem(M, Dout, sizeof(T));
  auto k = det_contract_kernel<T, DB>;
  gpk::allow_smem(k, sm);
  k<<<gpk::ceil_div(N, CR), CT, sm, st>>>(N, M, Dout, (const S*)kfu, lsf2, (const S*)A, (const S*)B, (S*)Bk,
                                          (S*)m_out, (S*)v_out);
}
template <typename T>
void contract_dispatch(int N, int M, int Dout, const void* kfu, const double* lsf2, const void* A, const void* B,
                       void* Bk, void* m_out, void* v_out, cudaStream_t st) {
  if (Dout == 1) contract_launch<T, 1>(N, M, Dout, kfu, lsf2, A, B, Bk, m_out, v_out, st);
  else if (Dout == 2) contract_launch<T, 2>(N, M, Dout, kfu, lsf2, A, B, Bk, m_out, v_out, st);
  else contract_launch<T, 4>(N, M, Dout, kfu, lsf2, A, B, Bk, m_out, v_out, st);
}
}  // namespace

// The sizes this entry point takes: M <= 128, and B and a few rows in the compute type within a CTA's shared memory, as
// det_contract_kernel lays them out.  (det_mma_kernel itself takes any Dout and M <= DM_MAX, and serves those
// through gpk_det_fwd.)
extern "C" int gpk_det_contract_supported(int prec, int M, int Dout) {
  const size_t tsz = prec == GPK_FP32 ? sizeof(float) : sizeof(df64);
  return M >= 1 && M <= 128 && Dout >= 1 && Dout <= DO_MAX && det_contract_smem(M, Dout, tsz) <= 227 * 1024;
}

extern "C" int gpk_det_contract(int prec, int N, int M, int Dout, const void* kfu, const double* lsf2, const void* A,
                                const void* B, int b_pairs, void* Bk, void* m_out, void* v_out, void* stream) {
  GPK_NVTX("gpk_det_contract");
  GPK_REQUIRE(prec == GPK_DF64 || prec == GPK_FP32, "det_contract: unknown precision %d", prec);
  GPK_REQUIRE(!b_pairs || prec == GPK_DF64, "det_contract: double-float pairs need GPK_DF64");
  GPK_REQUIRE(N >= 0 && M >= 1 && Dout >= 1, "det_contract: bad sizes N=%d M=%d Dout=%d", N, M, Dout);
  if (!gpk_det_contract_supported(prec, M, Dout))
    return gpk::fail(GPK_EUNSUPPORTED, "det_contract: M=%d, Dout=%d (needs M <= 128 and Dout M^2 in shared memory)",
                     M, Dout);
  GPK_REQUIRE(kfu && lsf2 && A && B, "det_contract: null input");
  if (N == 0) return GPK_OK;
  cudaStream_t st = gpk::as_stream(stream);
  if (prec == GPK_DF64)
    return dm_launch(N, M, Dout, lsf2, (const double*)A, (const double*)B, b_pairs, (const double*)kfu, (double*)Bk, (double*)m_out, (double*)v_out, st);
  contract_dispatch<float>(N, M, Dout, kfu, lsf2, A, B, Bk, m_out, v_out, st);
  return gpk::check_launch("det_contract");
}

extern "C" int gpk_det_bwd(int prec, int N, int M, int D, int Dout, const void* x, int ldx, const void* Z,
                           const double* lls2, const double* lsf2, const void* A, const void* kfu, const void* Bk,
                           const void* dm, const void* dv, const void* dkfu, double* dsf2, double* dl, double* dZ,
                           double* dA, void* dx, void* stream) {
  GPK_NVTX("gpk_det_bwd");
  return gpk_det_bwd_ws(prec, N, M, D, Dout, x, ldx, Z, lls2, lsf2, A, kfu, Bk, dm, dv, dkfu, dsf2, dl, dZ, dA, dx,
                        nullptr, 0, stream);
}

namespace {
// rows split over CTAs: threads are b (a multiple of 32 >= M) x row groups, 512 at most; CTAs of
// two passes of the row groups (8 rows at rg = 4): 125 CTAs for 1000 rows, one per SM at most
int det_bwd_grid(int N, int M) {
  const int bx = 32 * gpk::ceil_div(M, 32), rg = bx <= 128 ? 4 : 2;
  int grid = gpk::ceil_div(N, 2 * rg);
  if (grid > gpk::sm_count()) grid = gpk::sm_count();
  return grid;
}
long det_bwd_stride(int M, int D, int Dout, bool dkfu) { return (long)M * D + (long)(dkfu ? 0 : Dout) * M + 1 + D; }

// gram: 32 x 32 output tiles (the upper ones only when C is symmetric), rows split over
// gridDim.z chunks so that about two CTAs run per SM
int gram_chunks(int N, int M, bool sym) {
  const int nt = gpk::ceil_div(M, 32);
  const int tiles = sym ? nt * (nt + 1) / 2 : nt * nt;
  int chunks = gpk::ceil_div(gpk::sm_count() * 2, tiles);
  if (chunks > gpk::ceil_div(N, 16)) chunks = gpk::ceil_div(N, 16);
  if (chunks < 1) chunks = 1;
  return chunks;
}
}  // namespace

namespace {
template <typename T, int DC, int DB, bool EX>
void det_bwd_launch(int grid, dim3 threads, cudaStream_t st, int N, int M, int D, int Dout, const void* x, int ldx,
                    const void* Z, const double* lls2, const double* lsf2, const void* A, const void* kfu,
                    const void* Bk, const void* dm, const void* dv, const void* dkfu, double* dsf2, double* dl,
                    double* dZ, double* dA, void* dx, double* work, long stride) {
  typedef typename Num<T>::store_t S;
  const size_t sm = det_bwd_smem(threads.x, threads.y, DC, M, D, dkfu ? 0 : Dout, sizeof(T));
  auto k = det_bwd_kernel<T, DC, DB, EX>;
  gpk::allow_smem(k, sm);
  k<<<grid, threads, sm, st>>>(N, M, D, Dout, (const S*)x, ldx, (const S*)Z, lls2, lsf2, (const S*)A, (const S*)kfu,
                               (const S*)Bk, (const S*)dm, (const S*)dv, (const S*)dkfu, dsf2, dl, dZ, dA, (S*)dx,
                               work, stride);
}
// the exact forms for D = 8 inputs and 1 or 2 outputs given through A, Bk (the deep GP's first
// layer and the 8-input regressions); everything else takes the general form
template <typename T>
void det_bwd_dispatch(int grid, dim3 threads, cudaStream_t st, int dc, int N, int M, int D, int Dout, const void* x,
                      int ldx, const void* Z, const double* lls2, const double* lsf2, const void* A, const void* kfu,
                      const void* Bk, const void* dm, const void* dv, const void* dkfu, double* dsf2, double* dl,
                      double* dZ, double* dA, void* dx, double* work, long stride) {
#define GPK_DET_BWD_ARGS grid, threads, st, N, M, D, Dout, x, ldx, Z, lls2, lsf2, A, kfu, Bk, dm, dv, dkfu, dsf2, dl, \
                         dZ, dA, dx, work, stride
  if (D == 8 && !dkfu && Dout == 1) det_bwd_launch<T, 8, 1, true>(GPK_DET_BWD_ARGS);
  else if (D == 8 && !dkfu && Dout == 2) det_bwd_launch<T, 8, 2, true>(GPK_DET_BWD_ARGS);
  else if (dc == 8) det_bwd_launch<T, 8, DO_MAX, false>(GPK_DET_BWD_ARGS);
  else det_bwd_launch<T, 16, DO_MAX, false>(GPK_DET_BWD_ARGS);
#undef GPK_DET_BWD_ARGS
}
}  // namespace

long det_bwd_work_elems(int N, int M, int D, int Dout) {
  return (long)gpk::sm_count() * det_bwd_stride(M, D, Dout, false);
}
namespace {
// the pair-wise Gram reduction: pair blocks of GP_T * GP_PPT pairs, row chunks so that about one
// CTA runs per SM, each chunk at least 8 rows; rows staged GR at a time (about 48 KB)
int gram_pair_blocks(int M) { return gpk::ceil_div(M * (M + 1) / 2, GP_T * GP_PPT); }
int gram_pair_chunks(int N, int M) {
  int c = gpk::ceil_div(gpk::sm_count(), gram_pair_blocks(M));
  const int cap = gpk::ceil_div(N, 3);   // three rows a chunk or more (12 rows: 5.5 to 10.9 us at M = 5 to 200; eight: 5.8 to 11.3)
  if (c > cap) c = cap;
  return c < 1 ? 1 : c;
}
// the tensor-core form's split: rows a chunk (a multiple of 16) so that about one CTA runs per SM, tile
// groups of up to GM_TW tiles a warp (fewer where the chunks of 16 rows leave SMs idle: a tile's
// fold and float64 sums are then most of its time), k steps staged at a time; false where 16 rows of
// digits do not fit
struct GramMma {
  int groups, rows, chunks, ks, tw;
};
bool gram_mma_plan(int N, int M, int Dout, GramMma* g) {
  const size_t cap = 227 * 1024 - 64;
  if (gm_carve(nullptr, nullptr, M, 1) > cap) return false;
  const int tiles = gm_tiles(M), least = gpk::ceil_div(tiles, GM_W * GM_TW);
  const int want = std::max(1, gpk::sm_count() / (Dout * least));
  g->rows = 16 * std::max(1, gpk::ceil_div(gpk::ceil_div(N, want), 16));
  g->chunks = std::max(1, gpk::ceil_div(N, g->rows));
  g->tw = gpk::ceil_div(tiles, GM_W * std::max(least, std::min(tiles, gpk::sm_count() / (Dout * g->chunks))));
  g->groups = gpk::ceil_div(tiles, GM_W * g->tw);
  g->ks = std::min(8, g->rows / 16);
  while (gm_carve(nullptr, nullptr, M, g->ks) > cap) --g->ks;
  return true;
}
template <typename T, int DB>
void gram_pairs_launch(dim3 grid, size_t sm, cudaStream_t st, int N, int M, int Dout, const void* u, const void* w,
                       double* work, long pstride, int GR) {
  typedef typename Num<T>::store_t S;
  auto k = gram_pairs_kernel<T, DB>;
  gpk::allow_smem(k, sm);
  k<<<grid, GP_T, sm, st>>>(N, M, Dout, (const S*)u, (const S*)w, work, pstride, GR);
}
template <typename T>
void gram_pairs_dispatch(dim3 grid, size_t sm, cudaStream_t st, int N, int M, int Dout, const void* u, const void* w,
                         double* work, long pstride, int GR) {
  if (Dout == 1) gram_pairs_launch<T, 1>(grid, sm, st, N, M, Dout, u, w, work, pstride, GR);
  else if (Dout == 2) gram_pairs_launch<T, 2>(grid, sm, st, N, M, Dout, u, w, work, pstride, GR);
  else gram_pairs_launch<T, 4>(grid, sm, st, N, M, Dout, u, w, work, pstride, GR);
}

int gram_pair_rows(int M, size_t tsz) {
  const int r = (int)((48 * 1024) / ((size_t)M * tsz + DO_MAX * tsz));
  return r < 1 ? 1 : (r > 32 ? 32 : r);
}
}  // namespace

long gram_work_elems(int N, int M, int Dout) {
  const long full = (long)gram_chunks(N, M, false) * Dout * M * M;   // u != v: full tiles
  const long pairs = (long)gram_pair_chunks(N, M) * Dout * (M * (M + 1) / 2);
  GramMma g;
  // (a bound on chunks x Dout that grows with N and Dout: a workspace for the largest call serves smaller ones)
  long mma = 0;
  if (gram_mma_plan(N, M, Dout, &g)) {
    const long least = gpk::ceil_div(gm_tiles(M), GM_W * GM_TW);
    mma = std::min(std::max(gpk::sm_count() / least, (long)Dout), (long)Dout * std::max(1, gpk::ceil_div(N, 16))) *
          (M * (M + 1) / 2);
  }
  return std::max(full, std::max(pairs, mma));
}

extern "C" int gpk_det_bwd_ws(int prec, int N, int M, int D, int Dout, const void* x, int ldx, const void* Z,
                              const double* lls2, const double* lsf2, const void* A, const void* kfu, const void* Bk,
                              const void* dm, const void* dv, const void* dkfu, double* dsf2, double* dl, double* dZ,
                              double* dA, void* dx, double* work, long work_elems, void* stream) {
  GPK_NVTX("gpk_det_bwd_ws");
  GPK_REQUIRE(N >= 0 && M >= 1 && M <= 256 && D >= 1 && D <= 16, "det_bwd: bad sizes N=%d M=%d D=%d (M<=256, D<=16)", N, M, D);
  GPK_REQUIRE(dkfu || (Dout >= 1 && Dout <= DO_MAX), "det_bwd: Dout=%d outside [1,%d]", Dout, DO_MAX);
  GPK_REQUIRE(x && Z && lls2 && lsf2 && kfu && dsf2 && dl && dZ, "det_bwd: null");
  GPK_REQUIRE(dkfu || (A && Bk && dm && dv), "det_bwd: need dkfu or (A, Bk, dm, dv)");
  const long stride = det_bwd_stride(M, D, Dout, dkfu != nullptr);
  if (work) {
    const long need = (long)gpk::sm_count() * stride;
    GPK_REQUIRE(work_elems >= need, "det_bwd: workspace of %ld doubles, %ld needed", work_elems, need);
  }
  if (N == 0) return GPK_OK;
  cudaStream_t st = gpk::as_stream(stream);
  const int bx = 32 * gpk::ceil_div(M, 32), rg = bx <= 128 ? 4 : 2;
  const int grid = det_bwd_grid(N, M);
  const dim3 threads(bx, rg);
  const int dc = D <= 8 ? 8 : 16;
  if (prec == GPK_DF64)
    det_bwd_dispatch<df64>(grid, threads, st, dc, N, M, D, Dout, x, ldx, Z, lls2, lsf2, A, kfu, Bk, dm, dv, dkfu,
                           dsf2, dl, dZ, dA, dx, work, stride);
  else if (prec == GPK_FP32)
    det_bwd_dispatch<float>(grid, threads, st, dc, N, M, D, Dout, x, ldx, Z, lls2, lsf2, A, kfu, Bk, dm, dv, dkfu,
                            dsf2, dl, dZ, dA, dx, work, stride);
  else
    return gpk::fail(GPK_EINVAL, "det_bwd: unknown precision %d", prec);
  int rc = gpk::check_launch("det_bwd");
  if (rc != GPK_OK || !work) return rc;
  gpk::RedPlan plan{};
  plan.add(dZ, M * D);
  plan.add(dA, dkfu ? 0 : Dout * M);
  plan.add(dsf2, 1);
  plan.add(dl, D);
  return gpk::reduce_partials(work, grid, plan, st);
}

extern "C" int gpk_gram(int prec, int N, int M, int Dout, const void* u, const void* v, const void* w, double* C,
                        void* stream) {
  GPK_NVTX("gpk_gram");
  return gpk_gram_ws(prec, N, M, Dout, u, v, w, C, nullptr, 0, stream);
}

extern "C" int gpk_gram_ws(int prec, int N, int M, int Dout, const void* u, const void* v, const void* w, double* C,
                           double* work, long work_elems, void* stream) {
  GPK_NVTX("gpk_gram_ws");
  GPK_REQUIRE(N >= 0 && M >= 1 && Dout >= 1 && Dout <= DO_MAX, "gram: bad sizes");
  GPK_REQUIRE(u && v && w && C, "gram: null pointer");
  const int sym = u == v;   // C symmetric: the upper tiles only
  const int P = M * (M + 1) / 2;
  // the digits from a million pairs on: below, the tables and digits of a few rows a CTA take longer than the
  // double-float pairs (M = 100, one output: N = 128 9.9 us in pairs, 12.1 to 15.1 by digits; N = 256 12.8, 12.5 to
  // 15.1; N = 512 16.5, 14.6 to 17.7; M = 200: N = 64 14.9, 16.3 to 20.0; N = 128 19.0, 16.4 to 20.2)
  GramMma g{};
  const bool mma = prec == GPK_DF64 && sym && work && (long)N * P > GM_PAIRS && gram_mma_plan(N, M, Dout, &g);
  const int chunks = mma ? g.chunks : sym ? gram_pair_chunks(N, M) : gram_chunks(N, M, false);
  if (work) {
    const long need = (long)chunks * Dout * (sym ? P : M * M);
    GPK_REQUIRE(work_elems >= need, "gram: workspace of %ld doubles, %ld needed", work_elems, need);
  }
  if (N == 0) return GPK_OK;
  cudaStream_t st = gpk::as_stream(stream);
  if (sym && work) {   // the fixed-order symmetric form: unordered pairs, packed partial blocks
    const size_t tsz = prec == GPK_FP32 ? sizeof(float) : sizeof(df64);
    const int GR = gram_pair_rows(M, tsz);
    const size_t sm = (size_t)GR * (M + DO_MAX) * tsz;
    const dim3 grid(gram_pair_blocks(M), chunks);
    const long pstride = (long)Dout * P;
    if (mma) {
      const size_t smm = gm_carve(nullptr, nullptr, M, g.ks);
      gpk::allow_smem(gram_mma_kernel, smm);
      gram_mma_kernel<<<dim3(chunks, Dout, g.groups), GM_T, smm, st>>>(N, M, Dout, (const double*)u, (const double*)w,
                                                                       work, pstride, g.rows, g.ks, g.tw);
    } else if (prec == GPK_DF64) gram_pairs_dispatch<df64>(grid, sm, st, N, M, Dout, u, w, work, pstride, GR);
    else if (prec == GPK_FP32) gram_pairs_dispatch<float>(grid, sm, st, N, M, Dout, u, w, work, pstride, GR);
    else return gpk::fail(GPK_EINVAL, "gram: unknown precision %d", prec);
    int rc = gpk::check_launch("gram_pairs");
    if (rc != GPK_OK) return rc;
    gpk::RedPlan plan{};
    plan.add(C, Dout * P, 1, M);
    return gpk::reduce_partials(work, chunks, plan, st);
  }
  const int nt = gpk::ceil_div(M, 32);
  const int tchunks = gram_chunks(N, M, sym);   // the tiled form (atomic, or u != v)
  const int tiles = sym ? nt * (nt + 1) / 2 : nt * nt;
  const dim3 grid(sym ? tiles : nt, sym ? 1 : nt, tchunks);
  if (prec == GPK_DF64)
    gram_kernel<df64><<<grid, 256, 0, st>>>(N, M, Dout, (const double*)u, (const double*)v, (const double*)w, C,
                                            sym, work);
  else if (prec == GPK_FP32)
    gram_kernel<float><<<grid, 256, 0, st>>>(N, M, Dout, (const float*)u, (const float*)v, (const float*)w, C,
                                             sym, work);
  else
    return gpk::fail(GPK_EINVAL, "gram: unknown precision %d", prec);
  int rc = gpk::check_launch("gram");
  if (rc != GPK_OK || !work) return rc;
  gpk::RedPlan plan{};
  plan.add(C, Dout * M * M);
  return gpk::reduce_partials(work, tchunks, plan, st);
}

extern "C" int gpk_wsum(int prec, int N, int M, int Dout, const void* u, const void* w, double* c, void* stream) {
  GPK_NVTX("gpk_wsum");
  GPK_REQUIRE(N >= 0 && M >= 1 && Dout >= 1 && Dout <= DO_MAX, "wsum: bad sizes");
  GPK_REQUIRE(u && w && c, "wsum: null pointer");
  if (N == 0) return GPK_OK;
  cudaStream_t st = gpk::as_stream(stream);
  int gy = gpk::ceil_div(N, 8 * WU);
  if (gy > 128) gy = 128;
  dim3 grid(gpk::ceil_div(M, 32), gy);
  if (prec == GPK_DF64)
    wsum_kernel<df64><<<grid, 256, 0, st>>>(N, M, Dout, (const double*)u, (const double*)w, c);
  else if (prec == GPK_FP32)
    wsum_kernel<float><<<grid, 256, 0, st>>>(N, M, Dout, (const float*)u, (const float*)w, c);
  else
    return gpk::fail(GPK_EINVAL, "wsum: unknown precision %d", prec);
  return gpk::check_launch("wsum");
}

// the translation unit's bounds word (debug build; 0 otherwise)
GPK_BOUNDS_READER(kern)
