// Psi statistics of the ARD kernel under Gaussian inputs, fused with the
// moment-matching contractions of a sparse-GP layer, and their backward pass.
//
// Work decomposition (the general forward; the other kernels split it by warps): a CTA takes a contiguous range of data points, NPB
// points per pass; per pass its threads first build the points' tables in shared memory
// (per-dimension constants, per-pseudo-input terms u_a, h_aq), then sweep the M(M+1)/2
// unordered pairs (a <= b) of pseudo-inputs, each pair for all NPB points.  Each thread
// owns a fixed set of pairs (p = tid + k*NT) across all of its points, so sums over n of
// per-pair quantities (sum_n psi2, dB = sum_n dv psi2) stay in registers until one atomic
// flush per CTA.  psi2 per point is never materialised in HBM (unless requested).
//
// log2 psi2[n,a,b] = u_a + u_b + G_ab - sum_q t_aq t_bq   with
//   t_aq = (mu_q - z_aq) sqrt(c_q log2(e) / 2),  c_q = 1 / (l_q + 2 S_q)     (per point)
//   u_a  = k_n/2 - 1/2 sum_q t_aq^2                                         (per point)
//   k_n  = log2(e) (2 log sf2 + 1/2 sum_q log(l_q / (l_q + 2 S_q)))
//   G_ab = -log2(e) sum_q (z_aq - z_bq)^2 / (4 l_q)                          (per call)
// which is the reference's exponent (geepee/kernels.py:219-225) regrouped about the point, so
// that no term is larger than the exponent itself needs: where psi2 is not negligible,
// sum_q t_aq^2 < k_n + 127 (l + 2S >= l gives log2 psi2 <= k_n - sum_q (t_aq^2 + t_bq^2)).  In
// double-float precision u, t and G are therefore kept as fixed-point integers: the sums are
// integer additions, the cross terms 32 x 32 -> 64-bit multiply-adds, and the exponential reads
// its table index and remainder from the bits (exp2_fx).  Against double-float sums and exp_tab
// that is ~55 instead of ~140 instructions per pair and point for two dimensions; forward moments
// at N = 10000, Q = 5, M = 100: 498 -> 366 us.
//
// Template parameters: T compute type (df64 or float); PPT pairs per thread held in
// registers (0: plain strided sweep); QC a compile-time cap on Q and DB on Dout, so
// every per-dimension / per-output array is fully unrolled into registers.
#pragma once
#include "common.cuh"

namespace psi_impl {

constexpr int QMAX = 8;
constexpr int DMAX = 4;
constexpr int NT = 512;        // threads per CTA (forward)
// The widths: 2 (Q <= 2) and QMAX are the catch-all ones; 4 (Q = 3, 4) and 5 serve the plain forms only.
// At width QMAX, Q = 3 does nearly three times the row sums it needs: N = 5000, M = 90, Q = 3 took
// 158 + 409 us forward and backward there, 119 + 293 us at width 4; Q = 4 162 + 416 against
// 121 + 303.  Q is QC itself at width 5 (the
// psi-statistics workload's): the per-dimension loops then carry no runtime test.
__host__ __device__ constexpr bool exact_q(int QC) { return QC == 5; }
__host__ __device__ constexpr bool plain_q(int QC) { return QC == 4 || QC == 5; }
// a pseudo-input's record in a point's table: u, t_1 .. t_QC (zeros past Q), padded to an odd
// count so that the lanes of a warp (consecutive pseudo-inputs) read different banks
__host__ __device__ constexpr int rec_len(int QC) { return (1 + QC) | 1; }
constexpr int SMEM_STATIC = 128;               // the kernels' static words
constexpr size_t SMEM_CAP = 227 * 1024 - SMEM_STATIC;   // dynamic shared memory of a CTA beside them
constexpr int PPT_MAX = 16;    // pairs per thread for register-resident per-pair sums
constexpr int FRED = 16;        // reduction slots per warp: forward

template <typename S>
struct PsiArgs {
  int N, M, Q, Dout;
  const S* mu;
  const S* var;
  const S* Z;
  const double* lls2;
  const double* lsf2;
  const S* A;
  const S* B;
  S* psi1;
  S* psi2;
  double* psi2_sum;
  S* m_out;
  S* v_out;
  const S* m;
  const S* dm;
  const S* dv;
  const S* dpsi1;    // optional [N,M]: replaces dm_all A
  int chain;         // forward rollout: point n > 0 takes point n-1's (m, v) as its (mu, var)
  int bs_smem;       // symmetrised B staged in shared memory (set by the launcher)
  int g_smem;        // G_ab in shared memory (set by the launcher)
  long b_stride;     // != 0: B is per point (B + n*b_stride), dv treated as 1
  double* dsf2;
  double* dl;
  double* dZ;
  double* dA;
  double* dB;
  S* dmu;
  S* dvar;
  double* part;      // backward, fixed-order path: this CTA's partial sums at part + blockIdx.x *
                     // part_stride ([dB pairs D*P | dA D*M | dZ M*Q | dsf2 | dl Q]), no atomics
  long part_stride;
};

__device__ __forceinline__ void pair_of(int p, int& a, int& b) { tri_pair(p, a, b); }

// How a precision keeps the pair exponent's terms (log2 units): R a table element, arg() the
// exponent of a pair from the two records and G, ev() its exponential.
template <typename T>
struct PairExp;

// FP32: floats, and the hardware's base-2 exponential
template <>
struct PairExp<float> {
  typedef float R;
  static constexpr int TAB = 0;    // exp table entries in shared memory
  static __device__ __forceinline__ R u_of(float x) { return x; }
  static __device__ __forceinline__ R t_of(float x) { return x; }
  static __device__ __forceinline__ R g_of(float x) { return x; }
  template <int QC>
  static __device__ __forceinline__ R arg(saddr a, saddr b, R g) {
    R x = (ldsv<R>(a) + ldsv<R>(b)) + g;
#pragma unroll
    for (int q = 1; q <= QC; ++q) x = __fmaf_rn(-ldsv<R>(a + 4 * q), ldsv<R>(b + 4 * q), x);
    return x;
  }
  static __device__ __forceinline__ float ev(R x, saddr) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  }
  static __device__ __forceinline__ float ev_st(R x, saddr tab) { return ev(x, tab); }
};

// double-float: u and G in units of 2^-52; t as two words, t = high 2^-26 + low 2^-57 (|low| <= 2^30),
// so that t_a t_b in units of 2^-52 is the product of the high words plus the mixed products
// shifted by 31.  sum_q t_q^2 < 254 (see above) bounds the high words by 2^30 and a mixed sum over
// eight dimensions by 2^62.5.
template <>
struct PairExp<df64> {
  typedef long long R;
  static constexpr int TAB = kFxTab;
  static __device__ __forceinline__ R u_of(df64 x) { return fx52_of(x); }
  static __device__ __forceinline__ R t_of(df64 x) { return fx57_words_of(x); }
  // below -1024 every pair's psi2 is zero already (the other terms sum to less than 127); the
  // half step of exp2_fx enters here
  static __device__ __forceinline__ R g_of(df64 x) {
    return (x.hi > -1024.f ? fx52_of(x) : -(1024LL << 52)) + kFxHalf;
  }
  // a record whose pairs are all zero: u + u_b + G < -126 for every live b (u_b <= 63.5), and no
  // sum leaves the range of +-2048
  static __device__ __forceinline__ R dead_u() { return -(400LL << 52); }
  template <int QC>
  static __device__ __forceinline__ R arg(saddr a, saddr b, R g) {
    long long x = ldsv<R>(a) + ldsv<R>(b) + g;
    long long mid = 0;
    int2 ta[QC], tb[QC];
#pragma unroll
    for (int q = 0; q < QC; ++q) {
      ta[q] = lds_i2(a + 8 * (1 + q));   // (low, high) words of t
      tb[q] = lds_i2(b + 8 * (1 + q));
      mid = mad_wide(ta[q].y, tb[q].x, mid);
      mid = mad_wide(ta[q].x, tb[q].y, mid);
    }
    long long hi = mid >> 31;
#pragma unroll
    for (int q = 0; q < QC; ++q) hi = mad_wide(ta[q].y, tb[q].y, hi);
    x -= hi;
    return x;
  }
  static __device__ __forceinline__ df64 ev(R x, saddr tab) { return exp2_fx(x, tab); }
  // the same as a float64
  static __device__ __forceinline__ double ev_st(R x, saddr tab) { return exp2_fx_double(x, tab); }
};

template <typename T>
__device__ __forceinline__ void load_pair_table(float2* tab) {
  if (PairExp<T>::TAB) load_exp2_table(tab);
}
__host__ __device__ inline size_t pair_table_bytes(size_t tsz) { return tsz == 8 ? kFxTab * sizeof(float2) : 0; }

// The symmetrised weights of the packed pairs, Bs[d P + p] = B_d[a,b] + B_d[b,a] (a != b) or
// B_d[a,a].  B is read along its rows: the triangle at and below the diagonal by asynchronous copies
// into Bs, then the one above, four loads in flight a thread, each entry added where its mirror
// image lies (reading a pair's two entries together took a 32-byte sector per transposed entry).
template <typename T, int NTH>
__device__ void stage_sym_B(T* Bs, const typename Num<T>::store_t* B, int M, int D, int P) {
  typedef typename Num<T>::store_t S;
  constexpr int K = 4;
  for (int d = 0; d < D; ++d, B += (size_t)M * M, Bs += P) {
#pragma unroll 1
    for (int p = threadIdx.x; p < P; p += NTH) {
      int ia, ib;
      pair_of(p, ia, ib);
      async_copy(reinterpret_cast<S*>(Bs) + p, B + ia * M + ib);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll 1
    for (int p0 = threadIdx.x; p0 < P; p0 += K * NTH) {
      S x[K];
      int o[K];
      bool off[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int p = p0 + k * NTH;
        int ia = 0, ib = 0;
        if (p < P) pair_of(p, ia, ib);
        const int ja = M - 1 - ib, jb = M - 1 - ia;   // row jb, column ja >= jb: consecutive threads descend
        off[k] = ja != jb;
        o[k] = p < P ? ja * (ja + 1) / 2 + jb : -1;
        x[k] = p < P && off[k] ? B[jb * M + ja] : S(0);
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (o[k] >= 0) {
          T w = Num<T>::ld(reinterpret_cast<const S*>(Bs)[o[k]]);
          if (off[k]) w = add(w, Num<T>::ld(x[k]));
          Bs[o[k]] = w;
        }
      }
    }
  }
}

// CTA-wide sum of K values per thread (valid in warp 0) from the first nact warps: each warp reduces them in multi-value butterflies
// of eight (warp_sum_many; lane 4v then holds value c0 + v), lane i of warp 0 adds value i (and
// i + 32) over the warps in order and shuffles it to the warp.  Fixed order; K <= RED.
template <typename T, int K, int RED>
__device__ __forceinline__ void block_sum_many(T (&vals)[K], T* red, int nact) {
  static_assert(K <= RED, "K values per warp slot");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < nact) {
#pragma unroll
    for (int c0 = 0; c0 < K; c0 += 8) {
      T t[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) t[u] = c0 + u < K ? vals[c0 + u] : Num<T>::zero();
      warp_sum_many<8>(t);
      if ((lane & 3) == 0 && c0 + (lane >> 2) < K) red[warp * RED + c0 + (lane >> 2)] = t[0];
    }
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int c0 = 0; c0 < K; c0 += 32) {
      T s = Num<T>::zero();
      if (c0 + lane < K) {
        s = red[c0 + lane];
        for (int w = 1; w < nact; ++w) s = add(s, red[w * RED + c0 + lane]);
      }
#pragma unroll
      for (int i = c0; i < K && i < c0 + 32; ++i) vals[i] = shfl_idx(s, i - c0);
    }
  }
}

// Per-point tables of one data point n: per-dimension constants (pmu, pis1 = 1/(l+S),
// pc = 1/(l+2S), psq = sqrt(pc log2(e)/2), pld1/pld2 = 1/2 log(l/(l+S)), 1/2 log(l/(l+2S))) and
// the pseudo-inputs' records (u_a, t_aq).  The backward keeps one point's tables, the forward NPB
// points' side by side.
constexpr int PD = 6;   // arrays of QMAX per-dimension constants
template <typename T>
struct PointSlot {
  T* pmu;
  T* pis1;
  T* pc;
  T* psq;
  T* pld1;
  T* pld2;
  typename PairExp<T>::R* rec;   // [M][rec_len]
  __device__ __forceinline__ PointSlot(T* pd, typename PairExp<T>::R* r)
      : pmu(pd), pis1(pd + QMAX), pc(pd + 2 * QMAX), psq(pd + 3 * QMAX), pld1(pd + 4 * QMAX), pld2(pd + 5 * QMAX),
        rec(r) {}
};

// per-point constants for dimension q of point n
template <typename T, typename S, typename Tab>
__device__ __forceinline__ void dims_of(const PsiArgs<S>& a, const T* ell2, const T* lnl, const Tab& tab,
                                        const PointSlot<T>& ps, int n, int q, int part) {
  // a rollout reads the previous point's outputs (written before the pass's last barrier)
  const S* pmu = a.chain ? (n > 0 ? a.m_out + (size_t)(n - 1) * a.Q : a.mu) : a.mu + (size_t)n * a.Q;
  const S* pvar = a.chain ? (n > 0 ? a.v_out + (size_t)(n - 1) * a.Q : a.var) : a.var + (size_t)n * a.Q;
  // the four transcendental pieces of dimension q run on four threads (part 0..3)
  const T var = Num<T>::ld(pvar[q]);
  const T s = (part & 1) ? add(ell2[q], add(var, var)) : add(ell2[q], var);   // l+2S : l+S
  if (part == 0) {
    ps.pmu[q] = Num<T>::ld(pmu[q]);
    ps.pis1[q] = recip(s);
  } else if (part == 1) {
    const T c = recip(s);
    ps.pc[q] = c;
    ps.psq[q] = sqrt_(mul(c, scale2(log2e_of(c), -1)));
  } else if (part == 2) {
    ps.pld1[q] = scale2(sub(lnl[q], log_tab(s, tab)), -1);
  } else {
    ps.pld2[q] = scale2(sub(lnl[q], log_tab(s, tab)), -1);
  }
}

// The record of one pseudo-input at one point in fixed point: a dead record (zero for every
// pair) where k_n - sum_q t_q^2 < -127.5.  *flag is set where the fixed-point range does not hold
// and the point takes psi2_general: non-finite terms, k_n above 126, or l + 2S < l (a
// negative variance; the rounding of a zero one is tolerated), for which the bound on t fails.
template <int QC>
__device__ __forceinline__ void put_rec(long long* r, df64 k2, df64 s2, const df64* t, float ld2, int* flag) {
  const bool in = s2.hi < 1e38f && k2.hi < 63.f && k2.hi > -1e38f && ld2 < 1e-6f;   // false for NaN
  if (!in) *flag = 1;
  const bool live = in && 2.f * k2.hi - s2.hi >= -127.5f;
  r[0] = live ? PairExp<df64>::u_of(sub(k2, scale2(s2, -1))) : PairExp<df64>::dead_u();
#pragma unroll
  for (int q = 0; q < QC; ++q) r[1 + q] = live ? PairExp<df64>::t_of(t[q]) : 0;
}
template <int QC>
__device__ __forceinline__ void put_rec(float* r, float k2, float s2, const float* t, float, int*) {
  r[0] = k2 - 0.5f * s2;
#pragma unroll
  for (int q = 0; q < QC; ++q) r[1 + q] = t[q];
}

// per-pseudo-input terms of one point: psi1_a (returned) and the record (u_a, t_aq)
template <typename T, int QC, typename Tab>
__device__ __forceinline__ T rows_of(const T* z, T lsf, const Tab& tab, const PointSlot<T>& ps, int Q, int ia,
                                     int* flag) {
  T e1 = lsf, kap = lsf, s2 = Num<T>::zero();
  T t[QC];
  float ld2 = -1e30f;
#pragma unroll
  for (int q = 0; q < QC; ++q) {
    t[q] = Num<T>::zero();
    if (q < Q) {
      const T d = sub(ps.pmu[q], z[ia * Q + q]);
      e1 = add(e1, sub(ps.pld1[q], scale2(mul(mul(d, d), ps.pis1[q]), -1)));
      kap = add(kap, scale2(ps.pld2[q], -1));
      ld2 = fmax_nan(ld2, Num<T>::approx(ps.pld2[q]));
      t[q] = mul(d, ps.psq[q]);
      s2 = fma_(t[q], t[q], s2);
    }
  }
  put_rec<QC>(ps.rec + ia * rec_len(QC), mul(kap, log2e_of(kap)), s2, t, ld2, flag);
  return exp_tab(e1, tab);
}

// the per-point constants beside the arrays: log sf2 + sum pld1, k_n / 2 (log2 units), max pld2
constexpr int PDN = PD * QMAX + 4;
// point n's constants by one warp (4 Q <= 32 lanes), *flag cleared
template <typename T, typename S, typename Tab>
__device__ __forceinline__ void consts_of(const PsiArgs<S>& a, const T* ell2, const T* lnl, const Tab& tab, T lsf,
                                          const PointSlot<T>& ps, int n, int Q, int lane, int* flag) {
  T* pd = ps.pmu;
  if (lane < 4 * Q) dims_of<T, S>(a, ell2, lnl, tab, ps, n, lane >> 2, lane & 3);
  __syncwarp();
  if (lane == 0) {
    T c1 = lsf;
    for (int q = 0; q < Q; ++q) c1 = add(c1, ps.pld1[q]);
    pd[PD * QMAX] = c1;
  } else if (lane == 1) {
    T k = lsf;
    float ld2 = -1e30f;
    for (int q = 0; q < Q; ++q) {
      k = add(k, scale2(ps.pld2[q], -1));
      ld2 = fmax_nan(ld2, Num<T>::approx(ps.pld2[q]));
    }
    pd[PD * QMAX + 1] = mul(k, log2e_of(k));
    pd[PD * QMAX + 2] = Num<T>::c(ld2);
  } else if (lane == 2) {
    *flag = 0;
  }
}
// pseudo-input ia's record at the point, and its psi1 (z: its coordinates)
template <typename T, int QC, typename Tab>
__device__ __forceinline__ T row_of(const T* z, const Tab& tab, const PointSlot<T>& ps, int Q, int ia, int* flag) {
  const T* pd = ps.pmu;
  T e1 = pd[PD * QMAX], s2 = Num<T>::zero(), t[QC];
#pragma unroll
  for (int q = 0; q < QC; ++q) {
    t[q] = Num<T>::zero();
    if (q < Q) {
      const T d = sub(ps.pmu[q], z[q]);
      e1 = fma_(mul(d, d), scale2(neg(ps.pis1[q]), -1), e1);
      t[q] = mul(d, ps.psq[q]);
      s2 = fma_(t[q], t[q], s2);
    }
  }
  put_rec<QC>(ps.rec + ia * rec_len(QC), pd[PD * QMAX + 1], s2, t, Num<T>::approx(pd[PD * QMAX + 2]), flag);
  return exp_tab(e1, tab);
}

// psi2 of one pair outside the fixed-point range, from the point's constants and the two
// pseudo-inputs (df64 only; rare, so out of line)
template <typename T>
__device__ __noinline__ T psi2_general(const T* za, const T* zb, const T* pd, const T* inv4l, T lsf, int Q,
                                       const float2* tab) {
  const T *pmu = pd, *pc = pd + 2 * QMAX, *pld2 = pd + 5 * QMAX;
  T x = add(lsf, lsf);
  for (int q = 0; q < Q; ++q) {
    const T v = sub(pmu[q], scale2(add(za[q], zb[q]), -1)), d = sub(za[q], zb[q]);
    x = add(x, sub(pld2[q], add(mul(mul(v, v), pc[q]), mul(mul(d, d), inv4l[q]))));
  }
  return exp_pair(x, ExpTab{tab});
}

// barrier ID over NW warps of the CTA
template <int ID, int NW>
__device__ __forceinline__ void warps_sync() {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(NW * 32) : "memory");
}
__host__ __device__ constexpr int zlen(int QC) { return (QC + 1) & ~1; }   // a z row, padded to pairs
// G_ab (log2 units) of a pair from the pseudo-inputs
template <typename T, int QC>
__device__ __forceinline__ typename PairExp<T>::R pair_G(const T* za, const T* zb, const T* inv4l, int Q) {
  T g = Num<T>::zero();
#pragma unroll
  for (int q = 0; q < QC; ++q) {
    if (q < Q) {
      const T d = sub(za[q], zb[q]);
      g = fma_(mul(d, d), inv4l[q], g);
    }
  }
  return PairExp<T>::g_of(neg(mul(g, log2e_of(g))));
}

// The per-CTA pair tables by NW warps (the CTA's first): the pair table, G (where wanted) and the
// symmetrised weights Bs[d P + p] = B_d[a,b] + B_d[b,a] (half of that with `half`), B_d[a,a] on the
// diagonal.  B is read along its rows by asynchronous copies, the triangle at and below the
// diagonal into Bs, the one above into `tmp` ([P], e.g. G before it is formed), and converted
// from there; reading each pair's two entries together took a 32-byte sector per transposed entry
// (36 MB of L2 reads over 152 CTAs at M = 100).  The loops are kept rolled: this code runs
// once per CTA, and unrolled its instruction fetches took longer than its work.
template <typename T, int QC, int NW, int BAR>
__device__ __forceinline__ void stage_pairs(const T* z, const T* inv4l, int Q, int M, int P, int D,
                                         const typename Num<T>::store_t* B, bool half, unsigned short* pab,
                                         typename PairExp<T>::R* G, T* Bs, T* tmp) {
  typedef typename Num<T>::store_t S;
  constexpr int ZL = zlen(QC), NTH = NW * 32;
  const int tid = threadIdx.x;
  for (int d = 0; Bs && d < D; ++d, B += (size_t)M * M, Bs += P) {
#pragma unroll 1
    for (int p = tid; p < P; p += NTH) {
      int ia, ib;
      pair_of(p, ia, ib);
      if (pab && d == 0) pab[p] = (unsigned short)((ia << 8) | ib);
      const int ja = M - 1 - ib, jb = M - 1 - ia;   // row jb, column ja >= jb: consecutive threads descend
      async_copy(reinterpret_cast<S*>(Bs) + p, B + ia * M + ib);
      async_copy(reinterpret_cast<S*>(tmp) + ja * (ja + 1) / 2 + jb, B + jb * M + ja);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    warps_sync<BAR, NW>();
#pragma unroll 1
    for (int p = tid; p < P; p += NTH) {
      bool off;
      if (pab) {
        off = (pab[p] >> 8) != (pab[p] & 0xff);
      } else {
        int ia, ib;
        pair_of(p, ia, ib);
        off = ia != ib;
      }
      T w = Num<T>::ld(reinterpret_cast<const S*>(Bs)[p]);
      if (off) {
        w = add(w, Num<T>::ld(reinterpret_cast<const S*>(tmp)[p]));
        if (half) w = scale2(w, -1);
      }
      Bs[p] = w;
    }
    warps_sync<BAR, NW>();
  }
  const bool have = Bs && pab;
#pragma unroll 1
  for (int p = tid; p < P && (G || !have); p += NTH) {
    int ia, ib;
    if (have) {
      const int ab = pab[p];
      ia = ab >> 8;
      ib = ab & 0xff;
    } else {
      pair_of(p, ia, ib);
      if (pab) pab[p] = (unsigned short)((ia << 8) | ib);
    }
    if (G) G[p] = pair_G<T, QC>(z + ia * ZL, z + ib * ZL, inv4l, Q);
  }
}

// two consecutive elements in one access
__device__ __forceinline__ void lds_two(saddr p, df64& a, df64& b) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a.hi), "=f"(a.lo), "=f"(b.hi), "=f"(b.lo) : "r"(p));
}
__device__ __forceinline__ void lds_two(saddr p, long long& a, long long& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(p));
}
__device__ __forceinline__ void lds_two(saddr p, float& a, float& b) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(p));
}

// ---------------------------------------------------------------------------------
// Forward, general form (sum_n psi2, rollouts, psi2 together with moments, sizes whose tables do not
// fit): NPB points per pass.  Per pass: the NPB points' per-dimension constants (threads over
// (point, q)), then their per-pseudo-input terms (threads over (point, a)), then the pair
// sweep, in which each thread loads a pair's point-independent data once (G_ab, the symmetrised B
// weights) and evaluates psi2 for all NPB points, and finally one CTA reduction for the NPB
// points' m and v.  PPT > 0 keeps sum_n psi2 of each thread's pairs in registers (pairs
// tid + k*NT); PPT == 0 sweeps any number of pairs.
template <typename T>
struct FSmem {
  float2* tab;
  T* z;      // [M*Q]
  T* ell2;   // [QMAX]
  T* lnl;    // [QMAX]
  T* inv4l;  // [QMAX]
  T* misc;   // [4] log sf2, sf2
  T* pd;     // [NPB][PD][QMAX] per-point constants
  typename PairExp<T>::R* rec;   // [NPB][M][rec_len]
  T* p1;     // [NPB][M]
  T* As;     // [Dout][M]
  typename PairExp<T>::R* G;      // [P] or nullptr (then formed for each pair)
  T* Bs;     // [Dout*P] or nullptr
  T* red;    // [NT/32][FRED]
};

__host__ __device__ inline size_t fwd_smem_bytes(int M, int Q, int QC, int D, int npb, size_t tsz, int ng, int nbs) {
  size_t n = (size_t)M * Q + 3 * QMAX + 4 + (size_t)npb * PD * QMAX + (size_t)npb * M * (1 + rec_len(QC)) +
             (size_t)D * M + ng + nbs + (size_t)(NT / 32) * FRED;
  return pair_table_bytes(tsz) + n * tsz;
}

template <typename T, int QC>
__device__ FSmem<T> fcarve(char* base, int M, int Q, int D, int npb, int ng, int nbs) {
  typedef typename PairExp<T>::R R;
  static_assert(sizeof(R) == sizeof(T), "table elements as large as T");
  FSmem<T> s;
  s.tab = reinterpret_cast<float2*>(base);
  T* t = reinterpret_cast<T*>(base + pair_table_bytes(sizeof(T)));
  s.z = t; t += M * Q;
  s.ell2 = t; t += QMAX;
  s.lnl = t; t += QMAX;
  s.inv4l = t; t += QMAX;
  s.misc = t; t += 4;
  s.pd = t; t += npb * PD * QMAX;
  s.rec = reinterpret_cast<R*>(t); t += npb * M * rec_len(QC);
  s.p1 = t; t += npb * M;
  s.As = t; t += D * M;
  s.G = ng ? reinterpret_cast<R*>(t) : nullptr; t += ng;
  s.Bs = nbs ? t : nullptr; t += nbs;
  s.red = t;
  return s;
}

template <typename T, int NPB, int PPT, int QC, int DB>
__global__ void __launch_bounds__(NT) psi_fwd_gen_kernel(PsiArgs<typename Num<T>::store_t> a) {
  typedef typename Num<T>::store_t S;
  typedef PairExp<T> X;
  typedef typename X::R R;
  constexpr int RL = rec_len(QC);
  extern __shared__ __align__(16) char smem_raw[];
  const int M = a.M, Q = exact_q(QC) ? QC : a.Q, D = a.Dout;
  const int P = M * (M + 1) / 2;
  const bool contract = (a.A != nullptr) && (a.B != nullptr) && (a.m_out != nullptr || a.v_out != nullptr);
  FSmem<T> s = fcarve<T, QC>(smem_raw, M, Q, contract ? D : 0, NPB, a.g_smem ? P : 0, a.bs_smem ? D * P : 0);
  __shared__ int s_flag[NPB];   // a point of the pass lies outside the fixed-point range
  const ExpTab etab{s.tab};
  // ---- per-CTA tables: exp table, Z, lengthscales, sf2, A, G_ab and the symmetrised B
  load_pair_table<T>(s.tab);
  for (int i = threadIdx.x; i < M * Q; i += NT) s.z[i] = Num<T>::ld(a.Z[i]);
  if (contract)
    for (int i = threadIdx.x; i < D * M; i += NT) s.As[i] = Num<T>::ld(a.A[i]);
  __syncthreads();
  if (threadIdx.x < Q) {
    const int q = threadIdx.x;
    T lnl = Num<T>::ld(static_cast<S>(a.lls2[q]));
    T l2 = exp_tab(lnl, etab);
    s.lnl[q] = lnl;
    s.ell2[q] = l2;
    s.inv4l[q] = recip(mul(l2, Num<T>::c(4.f)));
  }
  if (threadIdx.x == 32) {
    T lsf = Num<T>::ld(static_cast<S>(a.lsf2[0]));
    s.misc[0] = lsf;
    s.misc[1] = exp_tab(lsf, etab);
  }
  __syncthreads();
  if (s.G) {
    for (int p = threadIdx.x; p < P; p += NT) {
      int ia, ib;
      pair_of(p, ia, ib);
      s.G[p] = pair_G<T, QC>(s.z + ia * Q, s.z + ib * Q, s.inv4l, Q);
    }
  }
  if (s.Bs) stage_sym_B<T, NT>(s.Bs, a.B, M, D, P);
  constexpr int KP = PPT > 0 ? PPT : 1;
  T acc[KP];
  int pab[KP];
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    acc[k] = Num<T>::zero();
    int p = threadIdx.x + k * NT, ia = 0, ib = 0;
    if (PPT > 0 && p < P) pair_of(p, ia, ib);
    pab[k] = (ia << 16) | ib;
  }
  __syncthreads();

  const T lsf = s.misc[0];
  // each CTA takes a contiguous range of points, NPB at a time
  const int nbeg = (int)((long)a.N * blockIdx.x / gridDim.x);
  const int nend = (int)((long)a.N * (blockIdx.x + 1) / gridDim.x);
  for (int n0 = nbeg; n0 < nend; n0 += NPB) {
    const int npts = min(NPB, nend - n0);
    auto slot = [&](int pt) { return PointSlot<T>(s.pd + pt * PD * QMAX, s.rec + pt * M * RL); };
    // ---- per-dimension constants of the NPB points
    if (threadIdx.x < NPB) s_flag[threadIdx.x] = 0;
    for (int t = threadIdx.x; t < 4 * npts * Q; t += NT) {
      const int part = t & 3, pq = t >> 2, pt = pq / Q, q = pq - pt * Q;
      dims_of<T, S>(a, s.ell2, s.lnl, etab, slot(pt), n0 + pt, q, part);
    }
    __syncthreads();
    // ---- per-pseudo-input terms (and psi1)
    for (int t = threadIdx.x; t < npts * M; t += NT) {
      const int pt = t / M, ia = t - pt * M;
      const T v1 = rows_of<T, QC>(s.z, lsf, etab, slot(pt), Q, ia, &s_flag[pt]);
      s.p1[pt * M + ia] = v1;
      if (a.psi1) a.psi1[(size_t)(n0 + pt) * M + ia] = Num<T>::st(v1);
    }
    __syncthreads();
    // ---- pairs
    bool any_flag = false;
    if (X::TAB) {
#pragma unroll
      for (int pt = 0; pt < NPB; ++pt) any_flag |= s_flag[pt] != 0;
    }
    T vacc[NPB][DB];
#pragma unroll
    for (int pt = 0; pt < NPB; ++pt)
#pragma unroll
      for (int d = 0; d < DB; ++d) vacc[pt][d] = Num<T>::zero();
    auto do_pair = [&](int p, int ia, int ib, T& sum) {
      const R gab = s.G ? s.G[p] : pair_G<T, QC>(s.z + ia * Q, s.z + ib * Q, s.inv4l, Q);
      T w[DB];
      if (contract) {
#pragma unroll
        for (int d = 0; d < DB; ++d) {
          w[d] = Num<T>::zero();
          if (d < D) {
            if (s.Bs) {
              w[d] = s.Bs[d * P + p];
            } else {
              const S* Bd = a.B + (size_t)d * M * M;
              w[d] = Num<T>::ld(Bd[ia * M + ib]);
              if (ia != ib) w[d] = add(w[d], Num<T>::ld(Bd[ib * M + ia]));
            }
          }
        }
      }
#pragma unroll
      for (int pt = 0; pt < NPB; ++pt) {
        if (pt < npts) {
          const R* rec = s.rec + pt * M * RL;
          const T ps = X::TAB && s_flag[pt] ? psi2_general(s.z + ia * Q, s.z + ib * Q, s.pd + pt * PD * QMAX, s.inv4l, lsf, Q, s.tab)
                               : X::ev(X::template arg<QC>(sm_addr(rec + ia * RL), sm_addr(rec + ib * RL), gab), sm_addr(s.tab));
          if (a.psi2) {
            const S v = Num<T>::st(ps);
            const size_t o = (size_t)(n0 + pt) * M;
            a.psi2[(o + ia) * M + ib] = v;
            a.psi2[(o + ib) * M + ia] = v;
          }
          if (PPT > 0) sum = add(sum, ps);
          if (contract) {
#pragma unroll
            for (int d = 0; d < DB; ++d)
              if (d < D) vacc[pt][d] = fma_(w[d], ps, vacc[pt][d]);
          }
        }
      }
    };
    if (PPT > 0) {
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        const int p = threadIdx.x + k * NT;
        if (p < P) do_pair(p, pab[k] >> 16, pab[k] & 0xffff, acc[k]);
      }
    } else if (contract && !a.psi2 && s.Bs && D == DB && !any_flag) {
      // moments only, every point in the fixed-point range: branch-free over the pass's slots, so that
      // their exps interleave (the steps of do_pair, so the same bits; a pass with fewer points
      // runs the extra slots on stale tables and never reads their sums).  N = 777, Q = 2, M = 200:
      // 151 -> 138 us
      constexpr int E = sizeof(T);
      const saddr ar = sm_addr(s.rec), at = sm_addr(s.tab), step = M * (RL * E);
      for (int p = threadIdx.x; p < P; p += NT) {
        int ia, ib;
        pair_of(p, ia, ib);
        const R gab = s.G ? s.G[p] : pair_G<T, QC>(s.z + ia * Q, s.z + ib * Q, s.inv4l, Q);
        T w[DB];
#pragma unroll
        for (int d = 0; d < DB; ++d) w[d] = s.Bs[d * P + p];
        saddr ra = ar + ia * (RL * E), rb = ar + ib * (RL * E);
        R arg[NPB];
#pragma unroll
        for (int pt = 0; pt < NPB; ++pt) {
          arg[pt] = X::template arg<QC>(ra, rb, gab);
          ra += step;
          rb += step;
        }
#pragma unroll
        for (int pt = 0; pt < NPB; ++pt) {
          const T ps = X::ev(arg[pt], at);
#pragma unroll
          for (int d = 0; d < DB; ++d) vacc[pt][d] = fma_(w[d], ps, vacc[pt][d]);
        }
      }
    } else {
      T dummy = Num<T>::zero();
      for (int p = threadIdx.x; p < P; p += NT) {
        int ia, ib;
        pair_of(p, ia, ib);
        do_pair(p, ia, ib, dummy);
      }
    }
    if (contract) {
      // m = psi1 . A_d per point, then one CTA reduction of (m, v) for the NPB points
      T vals[2 * NPB * DB];
#pragma unroll
      for (int pt = 0; pt < NPB; ++pt)
#pragma unroll
        for (int d = 0; d < DB; ++d) {
          T mm = Num<T>::zero();
          if (pt < npts && d < D)
            for (int ia = threadIdx.x; ia < M; ia += NT) mm = fma_(s.p1[pt * M + ia], s.As[d * M + ia], mm);
          vals[(pt * DB + d) * 2] = mm;
          vals[(pt * DB + d) * 2 + 1] = vacc[pt][d];
        }
      block_sum_many<T, 2 * NPB * DB, FRED>(vals, s.red, NT / 32);
      if (threadIdx.x == 0) {
#pragma unroll
        for (int pt = 0; pt < NPB; ++pt)
#pragma unroll
          for (int d = 0; d < DB; ++d) {
            if (pt < npts && d < D) {
              const int n = n0 + pt;
              const T mm = vals[(pt * DB + d) * 2];
              const T vv = sub(add(s.misc[1], vals[(pt * DB + d) * 2 + 1]), mul(mm, mm));
              if (a.m_out) a.m_out[(size_t)n * D + d] = Num<T>::st(mm);
              if (a.v_out) a.v_out[(size_t)n * D + d] = Num<T>::st(vv);
            }
          }
      }
    }
    __syncthreads();
  }
  if (PPT > 0 && a.psi2_sum) {
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      int p = threadIdx.x + k * NT;
      if (p < P) {
        int ia = pab[k] >> 16, ib = pab[k] & 0xffff;
        double v = (double)Num<T>::st(acc[k]);
        atomicAdd(&a.psi2_sum[ia * M + ib], v);
        if (ia != ib) atomicAdd(&a.psi2_sum[ib * M + ia], v);
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// Backward.  Per point: psi1 terms per pseudo-input; per pair L = W psi2 with
// W = sum_d dv_d (B_d[a,b] + B_d[b,a]) / 2 (the symmetrised upstream gradient, as psi2compDer does,
// geepee/kernels.py:415-418) staged in shared memory; then per row a the full-square sums
// R_a = sum_b L_ab, S_aq = sum_b L_ab z_bq.  With d_a = mu - z_a, A_a = S_a - z_a R_a,
// H_a = R_a d_a - A_a / 2 (sum_a A_a = 0, L being symmetric), every psi2 gradient follows:
//   dZ_aq += (1/l - c) A_a + 2 c R_a d_a
//   dmu_q  = -2 c sum_a R_a d_a,   dS_q = c sum_a (2 c d_a H_a - R_a)
//   dl_q  += ell (sum_a R_a / l + dS_q - sum_a z_a A_a / l^2)
// and with L1_a = dpsi1_a psi1_a, y = L1 d / (l + S) the psi1 ones:
//   dZ_aq += y,  dmu_q = -sum y,  2 dS_q = sum (y d - L1) / (l + S),  dl_q += ell (sum L1 / l + 2 dS_q)
// which restate psi2compDer and psi1compDer (geepee/kernels.py:355-378, 402-444) without their
// N x M x M temporaries.  Only dmu and the two parts of dS are reduced per point (3 Q values); every
// other sum stays with the thread of its row until the end.
//
// The CTA is split by warps into NS sweep, NB back and NF front warps, which work side by side:
//   stage A: sweep warps: pair sweep of point i -> L, dB-hat  | back warps: gradients of point i-1
//   stage B: sweep and back warps: row sums of point i (SEG threads a row)
//   through both: front warps: constants, psi1 terms and records of point i+1
// with one CTA barrier after each stage.  In one-role form (every warp doing each phase in
// turn, six barriers a point) the per-row phases kept 4 of 16 warps busy and the barriers were
// the largest stall.  Weights of each point's own (b_stride) are staged by the sweep warps at the start
// of stage A: fetched pair by pair inside the sweep, every pair waited for two loads (N = 301,
// M = 67, Q = 3, with the call: 138 -> 111 us; N = 1000, M = 100, Q = 4 204 -> 139).  Measured (df64, with the reduction of the partial blocks): N = 10000, Q = 5,
// M = 100: 1591 -> 766 us, 660 -> ~400 instructions a pair and point, 65% of issue slots; N = 1000,
// Q = 2, M = 100: 128 -> 84 us, of which ~35 us are per-CTA tables and the flush; N = 4999, Q = 2,
// M = 50, two outputs: 295 -> 128 us; FP32 at N = 10000: 416 -> 236 us.  Bound by instruction
// issue, half of it FP32 additions of the double-float sums.  Records alternate between two
// slots, the small per-point arrays between three.
// dZ's row sums in the back threads' registers: one row a thread, and room for them
__host__ __device__ constexpr bool bwd_dz_reg(int QC, int M, int nb) { return QC < QMAX && M <= nb * 32; }
template <typename T>
struct BSmem {
  typedef typename PairExp<T>::R R;
  float2* tab;
  T* z;      // [M][zlen]
  T* ell2;   // [QMAX]
  T* lnl;    // [QMAX]
  T* inv4l;  // [QMAX]
  T* il;     // [QMAX]
  T* misc;   // [4] log sf2, sf2
  T* pd;     // [3][PDN] per-point constants
  T* pg;     // [3][2*DMAX] dm_all, dv
  T* As;     // [Dout][M]
  R* rec;    // [2][M][rec_len]
  T* L1;     // [3][M]
  T* dz;     // [QC][M] where a back thread has several rows (else in its registers)
  T* gA;     // [Dout][M]
  T* rows;   // [SEG][1+QC][M]
  T* red;    // [back warps][3 QC + 2]
  T* L;      // [P]
  R* G;      // [P] or nullptr (then formed for each pair)
  T* Bs;     // [Dout*P] or nullptr
  T* accB;   // [Dout*P] or nullptr: sum over the CTA's points of dv psi2 (dBhat)
  unsigned short* pab;  // [P] or nullptr: the pairs (a << 8 | b)
};
struct BLayout {
  int seg, ng, nbs, nacc, pab;   // row segments, elements of G, B, dB-hat; pair table or not
};
template <typename T>
__host__ __device__ inline size_t bcarve(BSmem<T>* out, char* base, int M, int QC, int P, int D, int nb,
                                         const BLayout& lo) {
  typedef typename PairExp<T>::R R;
  static_assert(sizeof(R) == sizeof(T), "table elements as large as T");
  BSmem<T> s;
  size_t o = 0;
  auto take = [&](size_t n) {
    char* p = base + o;
    o += n;
    return p;
  };
  const size_t e = sizeof(T);
  s.tab = (float2*)take(PairExp<T>::TAB * sizeof(float2));
  s.z = (T*)take((size_t)zlen(QC) * M * e);   // (16-byte aligned: read in pairs)
  s.ell2 = (T*)take(QMAX * e);
  s.lnl = (T*)take(QMAX * e);
  s.inv4l = (T*)take(QMAX * e);
  s.il = (T*)take(QMAX * e);
  s.misc = (T*)take(4 * e);
  s.pd = (T*)take(3 * PDN * e);
  s.pg = (T*)take(3 * 2 * DMAX * e);
  s.As = (T*)take((size_t)D * M * e);
  s.rec = (R*)take(2 * (size_t)M * rec_len(QC) * e);
  s.L1 = (T*)take(3 * (size_t)M * e);
  s.dz = (T*)take(bwd_dz_reg(QC, M, nb) ? 0 : (size_t)QC * M * e);
  s.gA = (T*)take((size_t)D * M * e);
  s.rows = (T*)take((size_t)lo.seg * (1 + QC) * M * e);
  s.red = (T*)take((size_t)nb * (3 * QC + 2) * e);
  s.L = (T*)take((size_t)P * e);
  s.G = lo.ng ? (R*)take((size_t)lo.ng * e) : nullptr;
  s.Bs = lo.nbs ? (T*)take((size_t)lo.nbs * e) : nullptr;
  s.accB = lo.nacc ? (T*)take((size_t)lo.nacc * e) : nullptr;
  s.pab = lo.pab ? (unsigned short*)take((size_t)P * sizeof(unsigned short)) : nullptr;
  if (out) *out = s;
  return o;
}

template <typename T, int DB, int QC, int NS, int NB, int NF>
__global__ void __launch_bounds__((NS + NB + NF) * 32, NS < 12 ? 2 : 1)
    psi_bwd_kernel(PsiArgs<typename Num<T>::store_t> a, BLayout lo) {
  typedef typename Num<T>::store_t S;
  typedef PairExp<T> X;
  typedef typename X::R R;
  constexpr int RL = rec_len(QC), ZL = zlen(QC), NTH = (NS + NB + NF) * 32, NTS = NS * 32;
  extern __shared__ __align__(16) char smem_raw[];
  const int M = a.M, Q = exact_q(QC) ? QC : a.Q, D = a.Dout;
  const int P = M * (M + 1) / 2;
  BSmem<T> s;
  bcarve<T>(&s, smem_raw, M, QC, P, D, NB, lo);
  __shared__ int s_flag[3];   // the slot's point lies outside the fixed-point range
  const ExpTab etab{s.tab};
  const int tid = threadIdx.x, lane = tid & 31;
  const bool back_warp = tid >= NTS && tid < NTS + NB * 32, front_warp = tid >= NTS + NB * 32;
  // ---- per-CTA tables: exp table, Z, A, lengthscales, sf2
  load_pair_table<T>(s.tab);
#pragma unroll 1
  for (int i = tid; i < M * ZL; i += NTH) {
    const int ia = i / ZL, q = i - ia * ZL;
    s.z[i] = q < Q ? Num<T>::ld(a.Z[ia * Q + q]) : Num<T>::zero();
  }
  const bool dz_reg = bwd_dz_reg(QC, M, NB);
  if (!dz_reg)
    for (int i = tid; i < M * QC; i += NTH) s.dz[i] = Num<T>::zero();
#pragma unroll 1
  for (int i = tid; i < D * M; i += NTH) {
    s.As[i] = a.dpsi1 ? Num<T>::zero() : Num<T>::ld(a.A[i]);
    s.gA[i] = Num<T>::zero();
  }
  double* const part = a.part ? a.part + (size_t)blockIdx.x * a.part_stride : nullptr;
  __syncthreads();
  if (tid < Q) {
    const T lnl = Num<T>::ld(static_cast<S>(a.lls2[tid]));
    const T l2 = exp_tab(lnl, etab);
    s.lnl[tid] = lnl;
    s.ell2[tid] = l2;
    s.il[tid] = recip(l2);
    s.inv4l[tid] = recip(mul(l2, Num<T>::c(4.f)));
  }
  if (tid == 32) {
    const T lsf = Num<T>::ld(static_cast<S>(a.lsf2[0]));
    s.misc[0] = lsf;
    s.misc[1] = exp_tab(lsf, etab);
  }
  __syncthreads();
  const T lsf = s.misc[0];
  // each CTA takes a contiguous range of points
  const int nbeg = (int)((long)a.N * blockIdx.x / gridDim.x);
  const int nend = (int)((long)a.N * (blockIdx.x + 1) / gridDim.x);
  const int cnt = nend - nbeg;

  // ---- front warps: constants, psi1 terms and records of point i
  auto front = [&](int i) {
    const int rt = tid - (NTS + NB * 32), rw = rt >> 5;
    const int n = nbeg + i, sl = i % 3;
    const PointSlot<T> ps(s.pd + sl * PDN, s.rec + (size_t)(i & 1) * M * RL);
    T* pg = s.pg + sl * 2 * DMAX;
    if (rw == 0) {
      consts_of<T, S>(a, s.ell2, s.lnl, etab, lsf, ps, n, Q, lane, &s_flag[sl]);
    } else if (rw == 1 && lane < D) {
      const T dvv = a.b_stride ? Num<T>::c(1.f) : Num<T>::ld(a.dv[(size_t)n * D + lane]);
      if (!a.dpsi1) {
        const T mm = Num<T>::ld(a.m[(size_t)n * D + lane]);
        const T dmv = Num<T>::ld(a.dm[(size_t)n * D + lane]);
        pg[lane] = sub(dmv, mul(scale2(dvv, 1), mm));     // dm_all
      }
      pg[DMAX + lane] = dvv;
    }
    warps_sync<2, NF>();
    for (int ia = rt; ia < M; ia += NF * 32) {
      const T p1 = row_of<T, QC>(s.z + ia * ZL, etab, ps, Q, ia, &s_flag[sl]);
      T dp1 = Num<T>::zero();
      if (a.dpsi1) {
        dp1 = Num<T>::ld(a.dpsi1[(size_t)n * M + ia]);
      } else {
#pragma unroll
        for (int d = 0; d < DB; ++d) {
          if (d < D) {
            dp1 = fma_(pg[d], s.As[d * M + ia], dp1);
            s.gA[d * M + ia] = fma_(pg[d], p1, s.gA[d * M + ia]);
          }
        }
      }
      s.L1[sl * M + ia] = mul(dp1, p1);
    }
    warps_sync<2, NF>();   // (the constants' slot is written again three points later)
  };

  // ---- back warps: gradients of point i from its row sums
  T g1 = Num<T>::zero(), g2 = Num<T>::zero();   // sum L1, sum R
  T dzr[QC];                                    // this thread's row of dZ (dz_reg)
  T g_z[QC], g_l = Num<T>::zero();              // sum z A; lane QC + q of the first back warp: sum (2 dS1 + dS2)
#pragma unroll
  for (int q = 0; q < QC; ++q) g_z[q] = dzr[q] = Num<T>::zero();
  constexpr int RW = 3 * QC + 2;
  auto back = [&](int i) {
    const int rt = tid - NTS, rw = rt >> 5;
    const int n = nbeg + i, sl = i % 3;
    const PointSlot<T> ps(s.pd + sl * PDN, s.rec);
    T tot = Num<T>::zero();
    for (int r0 = 0; r0 < M; r0 += NB * 32) {
      const int ia = r0 + rt;
      T vals[3 * QC];   // per dimension: -dmu, 2 dS of psi1, dS of psi2
#pragma unroll
      for (int k = 0; k < 3 * QC; ++k) vals[k] = Num<T>::zero();
      if (ia < M) {
        const T L1 = s.L1[sl * M + ia];
        const T* row = s.rows + ia;
        T Ra = row[0], Sa[QC];
#pragma unroll
        for (int q = 0; q < QC; ++q) Sa[q] = row[(1 + q) * M];
        for (int g = 1; g < lo.seg; ++g) {
          row += (1 + QC) * M;
          acc_add(Ra, row[0]);
#pragma unroll
          for (int q = 0; q < QC; ++q) acc_add(Sa[q], row[(1 + q) * M]);
        }
        Ra = acc_done(Ra);
        g1 = add(g1, L1);
        g2 = add(g2, Ra);
#pragma unroll
        for (int q = 0; q < QC; ++q) {
          if (q < Q) {
            const T z = s.z[ia * ZL + q], d = sub(ps.pmu[q], z), is1 = ps.pis1[q], c = ps.pc[q];
            const T y = mul(is1, mul(L1, d));
            const T A = sub(acc_done(Sa[q]), mul(Ra, z)), Rd = mul(Ra, d);
            const T yg = add(y, mul(scale2(c, 1), Rd));
            const T dz = fma_(sub(s.il[q], c), A, add(dz_reg ? dzr[q] : s.dz[q * M + ia], yg));
            if (dz_reg) dzr[q] = dz;
            else s.dz[q * M + ia] = dz;
            g_z[q] = fma_(z, A, g_z[q]);
            const T H = sub(Rd, scale2(A, -1));
            vals[q] = yg;
            vals[QC + q] = mul(is1, sub(mul(y, d), L1));
            vals[2 * QC + q] = mul(c, sub(scale2(mul(c, mul(d, H)), 1), Ra));
          }
        }
      }
      // 3 Q values over the back warps: multi-value butterflies, then lane k adds value k over warps
#pragma unroll
      for (int c0 = 0; c0 < 3 * QC; c0 += 8) {
        T t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) t[u] = c0 + u < 3 * QC ? vals[c0 + u] : Num<T>::zero();
        warp_sum_many<8>(t);
        if ((lane & 3) == 0 && c0 + (lane >> 2) < 3 * QC) s.red[rw * RW + c0 + (lane >> 2)] = t[0];
      }
      warps_sync<1, NB>();
      if (rw == 0 && lane < 3 * QC)
        for (int w = 0; w < NB; ++w) tot = add(tot, s.red[w * RW + lane]);
      warps_sync<1, NB>();   // red and the constants' slot are free again
    }
    if (rw == 0) {
      const T e2 = shfl_idx(tot, lane + QC);
      const int q = lane < QC ? lane : lane - QC;
      if (lane < 2 * QC && q < Q) {
        if (lane < QC) {
          a.dmu[(size_t)n * Q + q] = Num<T>::st(neg(tot));
        } else {
          a.dvar[(size_t)n * Q + q] = Num<T>::st(add(scale2(tot, -1), e2));
          g_l = add(g_l, add(tot, e2));
        }
      }
    }
  };

  if (front_warp) {
    if (cnt > 0) front(0);
  } else {
    constexpr int NTA = NTS + NB * 32;
    stage_pairs<T, QC, NS + NB, 3>(s.z, s.inv4l, Q, M, P, D, a.B, true, s.pab, s.G, a.b_stride ? nullptr : s.Bs, s.L);
    if (s.accB)
#pragma unroll 1
      for (int i = tid; i < D * P; i += NTA) s.accB[i] = Num<T>::zero();
    else if (part && a.dB)   // dBhat accumulates in this CTA's partial block (each pair has one owner)
      for (int i = tid; i < D * P; i += NTA) part[i] = 0.0;
  }
  __syncthreads();
  for (int i = 0; i < cnt; ++i) {
    const int n = nbeg + i, sl = i % 3;
    // ---- stage A
    if (front_warp) {
      if (i + 1 < cnt) front(i + 1);
    } else if (back_warp) {
      if (i > 0) back(i - 1);
    } else {
      const R* rec = s.rec + (size_t)(i & 1) * M * RL;
      const bool general = X::TAB && s_flag[sl];
      if (a.b_stride && s.Bs)   // this point's weights (the row sums of the last one are done with L)
        stage_pairs<T, QC, NS, 4>(s.z, s.inv4l, Q, M, P, 1, a.B + (size_t)n * a.b_stride, true, s.pab, nullptr, s.Bs, s.L);
      T dvr[DB];
#pragma unroll
      for (int d = 0; d < DB; ++d) dvr[d] = d < D ? s.pg[sl * 2 * DMAX + DMAX + d] : Num<T>::zero();
      if (D == DB && s.Bs && (s.accB || !a.dB) && s.G && s.pab && !general) {
        // the common configuration, branch-free: two pairs (p, p + NTS) per iteration, each step
        // written for both, so that their dependent chains interleave
        constexpr int E = sizeof(T);
        const bool sum = s.accB;
        const saddr ar = sm_addr(rec), aG = sm_addr(s.G), aB = sm_addr(s.Bs), aL = sm_addr(s.L),
                    aC = sum ? sm_addr(s.accB) : 0u, ap = sm_addr(s.pab), at = sm_addr(s.tab);
        for (int p0 = tid; p0 < P; p0 += 2 * NTS) {
          saddr o[2];   // the pairs' byte offsets
          R arg[2];
          const bool two = p0 + NTS < P;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int p = GPK_IDX(u && two ? p0 + NTS : p0, P, 2), ab = lds_u16(ap + 2 * p);
            o[u] = p * E;
            arg[u] = X::template arg<QC>(ar + (ab >> 8) * (RL * E), ar + (ab & 0xff) * (RL * E), ldsv<R>(aG + o[u]));
          }
          T ps2[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) ps2[u] = X::ev(arg[u], at);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            T ab[DB];
#pragma unroll
            for (int d = 0; d < DB; ++d) ab[d] = mul(dvr[d], ps2[u]);
            T l;
            if (DB == 1) {   // (dv psi2) B, reusing the dB-hat term
              l = mul(ab[0], ldsv<T>(aB + o[u]));
            } else {
              T w = mul(dvr[0], ldsv<T>(aB + o[u]));
#pragma unroll
              for (int d = 1; d < DB; ++d) w = fma_(dvr[d], ldsv<T>(aB + d * P * E + o[u]), w);
              l = mul(w, ps2[u]);
            }
            if (u == 0 || two) {
              sts(aL + o[u], l);
#pragma unroll
              for (int d = 0; d < DB; ++d)
                if (sum) sts(aC + d * P * E + o[u], add(ldsv<T>(aC + d * P * E + o[u]), ab[d]));
            }
          }
        }
      } else {
        for (int p = tid; p < P; p += NTS) {
          int ia, ib;
          pair_of(p, ia, ib);
          T ps2;
          if (general) {
            ps2 = psi2_general(s.z + ia * ZL, s.z + ib * ZL, s.pd + sl * PDN, s.inv4l, lsf, Q, s.tab);
          } else {
            const R gab = s.G ? s.G[p] : pair_G<T, QC>(s.z + ia * ZL, s.z + ib * ZL, s.inv4l, Q);
            ps2 = X::ev(X::template arg<QC>(sm_addr(rec + ia * RL), sm_addr(rec + ib * RL), gab), sm_addr(s.tab));
          }
          T w = Num<T>::zero();
#pragma unroll
          for (int d = 0; d < DB; ++d) {
            if (d < D) {
              T bb;
              if (s.Bs) {
                bb = s.Bs[d * P + p];
              } else {
                const S* Bd = a.B + (size_t)d * M * M + (size_t)n * a.b_stride;
                bb = Num<T>::ld(Bd[ia * M + ib]);
                if (ia != ib) bb = scale2(add(bb, Num<T>::ld(Bd[ib * M + ia])), -1);
              }
              w = fma_(dvr[d], bb, w);
            }
          }
          s.L[p] = mul(w, ps2);
#pragma unroll
          for (int d = 0; d < DB; ++d) {
            if (d < D) {
              const T ab = mul(dvr[d], ps2);
              if (s.accB) {
                s.accB[d * P + p] = add(s.accB[d * P + p], ab);
              } else if (part && a.dB) {   // no room for the accumulators: this thread's pair of the partial block
                part[d * P + p] += (double)Num<T>::st(ab);
              } else if (a.dB) {   // no room for the accumulators: straight into dB
                const double v = (double)Num<T>::st(ab);
                atomicAdd(&a.dB[((size_t)d * M + ia) * M + ib], v);
                if (ia != ib) atomicAdd(&a.dB[((size_t)d * M + ib) * M + ia], v);
              }
            }
          }
        }
      }
    }
    if (!front_warp) {
      warps_sync<3, NS + NB>();
      // ---- stage B: thread (segment, row) sums the row's columns [b0, b1) of the symmetric L;
      // lanes take consecutive rows, so z_b is one broadcast
      const int W = (M + lo.seg - 1) / lo.seg;
      for (int t = tid; t < lo.seg * M; t += NTS + NB * 32) {
        const int g = t / M, ia = t - g * M;
        const int b0 = g * W, b1 = min(M, b0 + W);
        constexpr int E = sizeof(T);
        saddr l = sm_addr(s.L) + (ia >= b0 ? ia * (ia + 1) / 2 + b0 : b0 * (b0 + 1) / 2 + ia) * E;
        saddr zb = sm_addr(s.z) + b0 * (ZL * E);
        T Rs = Num<T>::zero(), Sq[ZL];
#pragma unroll
        for (int q = 0; q < ZL; ++q) Sq[q] = Num<T>::zero();
#pragma unroll 4
        for (int b = b0; b < b1; ++b) {
          const T lv = ldsv<T>(l);
          l += b < ia ? E : (b + 1) * E;   // the next column of this row in the packed triangle
          acc_add(Rs, lv);
#pragma unroll
          for (int q = 0; q < ZL; q += 2) {
            T z0, z1;
            lds_two(zb + q * E, z0, z1);
            acc_fma(Sq[q], lv, z0);
            if (q + 1 < QC) acc_fma(Sq[q + 1], lv, z1);
          }
          zb += ZL * E;
        }
        T* o = s.rows + (size_t)g * (1 + QC) * M + ia;
        o[0] = acc_done(Rs);
#pragma unroll
        for (int q = 0; q < QC; ++q) o[(1 + q) * M] = acc_done(Sq[q]);
      }
    }
    __syncthreads();
  }
  if (back_warp && cnt > 0) back(cnt - 1);
  T* const dzo = dz_reg ? s.rows : s.dz;   // (a back thread has read its own column of rows)
  if (back_warp && dz_reg && tid - NTS < M) {
#pragma unroll
    for (int q = 0; q < QC; ++q)
      if (q < Q) dzo[q * M + tid - NTS] = dzr[q];
  }
  __syncthreads();
  // ---- flush CTA accumulators: into the partial block ([dB pairs D*P | dA D*M | dZ M*Q | dsf2 |
  // dl Q], fixed-order path) or atomically
  if (part) {
    const bool wantA = a.dA && !a.dpsi1;
    if (s.accB)
#pragma unroll 1
      for (int i = tid; i < D * P; i += NTH) part[i] = st_int(s.accB[i]);
#pragma unroll 1
    for (int i = tid; i < D * M; i += NTH) part[D * P + i] = wantA ? st_int(s.gA[i]) : 0.0;
#pragma unroll 1
    for (int i = tid; i < M * Q; i += NTH) {
      const int ia = i / Q, q = i - ia * Q;
      part[D * P + D * M + i] = st_int(dzo[q * M + ia]);
    }
  } else {
    if (a.dB && s.accB) {
      for (int p = tid; p < P; p += NTH) {
        int ia, ib;
        pair_of(p, ia, ib);
        for (int d = 0; d < D; ++d) {
          const double v = (double)Num<T>::st(s.accB[d * P + p]);
          atomicAdd(&a.dB[((size_t)d * M + ia) * M + ib], v);
          if (ia != ib) atomicAdd(&a.dB[((size_t)d * M + ib) * M + ia], v);
        }
      }
    }
    if (a.dA && !a.dpsi1)
      for (int i = tid; i < D * M; i += NTH) atomicAdd(&a.dA[i], (double)Num<T>::st(s.gA[i]));
    for (int i = tid; i < M * Q; i += NTH) {
      const int ia = i / Q, q = i - ia * Q;
      atomicAdd(&a.dZ[i], (double)Num<T>::st(dzo[q * M + ia]));
    }
  }
  // dsf2 and dl: (sum L1 + 2 sum R) / sf2 and ell ((sum L1 + sum R) / l + g_l - g_z / l^2)
  if (back_warp) {
    const int rt = tid - NTS, rw = rt >> 5;
    auto put = [&](int k, T v) {
      v = warp_sum(v);
      if (lane == 0) s.red[rw * RW + k] = v;
    };
    put(0, g1);
    put(1, g2);
#pragma unroll
    for (int q = 0; q < QC; ++q) put(2 + q, g_z[q]);
    if (rw == 0 && lane >= QC && lane < 2 * QC) s.red[2 + lane] = g_l;   // value 2 + QC + q
    warps_sync<1, NB>();
    if (rt < 1 + Q) {
      auto tot = [&](int k) {
        T v = s.red[k];
        for (int w = 1; w < NB; ++w) v = add(v, s.red[w * RW + k]);
        return v;
      };
      const T t1 = tot(0), t2 = tot(1);
      double out;
      if (rt == 0) {
        out = (double)Num<T>::st(div(add(t1, scale2(t2, 1)), s.misc[1]));
      } else {
        const int q = rt - 1;
        const T il = s.il[q];
        const T g = add(mul(add(t1, t2), il), sub(s.red[2 + QC + q], mul(tot(2 + q), mul(il, il))));
        out = (double)Num<T>::st(mul(g, sqrt_(s.ell2[q])));
      }
      if (part) part[D * P + D * M + M * Q + rt] = out;
      else atomicAdd(rt == 0 ? a.dsf2 : a.dl + (rt - 1), out);
    }
  }
}

// ---------------------------------------------------------------------------------
// Forward moments (m, v and optionally psi1), NPB points per pass, split by warps like the backward:
// NS sweep warps take the pairs of pass i (each thread a pair for all NPB points, G and B loaded
// once) while NF front warps form the constants, psi1, m and the records of pass i + 1 and finish
// pass i - 1's v from the sweep warps' sums: one CTA barrier a pass.  Measured (df64), general form
// of the same sweep -> this: N = 10000, Q = 5, M = 100: 366 -> 285 us (64% of issue slots; 143
// instructions a pair and point); N = 1000, Q = 2: 50 -> 41 us, of which ~18 us are the per-CTA
// tables; N = 4999, Q = 2, M = 50, two outputs: 85 -> 62 us.
template <typename T>
struct MSmem {
  typedef typename PairExp<T>::R R;
  float2* tab;
  T* z;      // [M][zlen]
  T* ell2;   // [QMAX]
  T* lnl;    // [QMAX]
  T* inv4l;  // [QMAX]
  T* misc;   // [4] log sf2, sf2
  T* pd;     // [2][NPB][PDN] per-point constants
  T* As;     // [Dout][M]
  T* p1;     // [NPB][M]
  T* ms;     // [3][NPB][DMAX] m of three passes
  T* red;    // [2][NS][NPB*DB]
  R* rec;    // [2][NPB][M][rec_len]
  R* G;      // [P]
  T* Bs;     // [Dout*P]
  unsigned short* pab;   // [P] or nullptr
};
template <typename T>
__host__ __device__ inline size_t mcarve(MSmem<T>* out, char* base, int M, int QC, int P, int D, int npb, int ns,
                                         int db, int pab) {
  typedef typename PairExp<T>::R R;
  MSmem<T> s;
  size_t o = 0;
  auto take = [&](size_t n) {
    char* p = base + o;
    o += n;
    return p;
  };
  const size_t e = sizeof(T);
  s.tab = (float2*)take(PairExp<T>::TAB * sizeof(float2));
  s.z = (T*)take((size_t)zlen(QC) * M * e);
  s.ell2 = (T*)take(QMAX * e);
  s.lnl = (T*)take(QMAX * e);
  s.inv4l = (T*)take(QMAX * e);
  s.misc = (T*)take(4 * e);
  s.pd = (T*)take((size_t)2 * npb * PDN * e);
  s.As = (T*)take((size_t)D * M * e);
  s.p1 = (T*)take((size_t)npb * M * e);
  s.ms = (T*)take((size_t)3 * npb * DMAX * e);
  s.red = (T*)take((size_t)2 * ns * npb * db * e);
  s.rec = (R*)take((size_t)2 * npb * M * rec_len(QC) * e);
  s.G = (R*)take((size_t)P * e);
  s.Bs = (T*)take((size_t)D * P * e);
  s.pab = pab ? (unsigned short*)take((size_t)P * sizeof(unsigned short)) : nullptr;
  if (out) *out = s;
  return o;
}

template <typename T, int NPB, int QC, int DB, int NS, int NF>
__global__ void __launch_bounds__((NS + NF) * 32, NS < 16 ? 2 : 1)
    psi_fwd_kernel(PsiArgs<typename Num<T>::store_t> a, int use_pab) {
  typedef typename Num<T>::store_t S;
  typedef PairExp<T> X;
  typedef typename X::R R;
  constexpr int RL = rec_len(QC), ZL = zlen(QC), NTH = (NS + NF) * 32, NTS = NS * 32, K = NPB * DB;
  static_assert(K <= 8, "one butterfly of eight values");
  extern __shared__ __align__(16) char smem_raw[];
  const int M = a.M, Q = exact_q(QC) ? QC : a.Q, D = a.Dout;
  const int P = M * (M + 1) / 2;
  MSmem<T> s;
  mcarve<T>(&s, smem_raw, M, QC, P, D, NPB, NS, DB, use_pab);
  __shared__ int s_flag[2][NPB];   // a point of the pass lies outside the fixed-point range
  const ExpTab etab{s.tab};
  const int tid = threadIdx.x, lane = tid & 31;
  const bool front_warp = tid >= NTS;
  // ---- per-CTA tables
  load_pair_table<T>(s.tab);
#pragma unroll 1
  for (int i = tid; i < M * ZL; i += NTH) {
    const int ia = i / ZL, q = i - ia * ZL;
    s.z[i] = q < Q ? Num<T>::ld(a.Z[ia * Q + q]) : Num<T>::zero();
  }
#pragma unroll 1
  for (int i = tid; i < D * M; i += NTH) s.As[i] = Num<T>::ld(a.A[i]);
  __syncthreads();
  if (tid < Q) {
    const T lnl = Num<T>::ld(static_cast<S>(a.lls2[tid]));
    const T l2 = exp_tab(lnl, etab);
    s.lnl[tid] = lnl;
    s.ell2[tid] = l2;
    s.inv4l[tid] = recip(mul(l2, Num<T>::c(4.f)));
  }
  if (tid == 32) {
    const T lsf = Num<T>::ld(static_cast<S>(a.lsf2[0]));
    s.misc[0] = lsf;
    s.misc[1] = exp_tab(lsf, etab);
  }
  __syncthreads();
  const T lsf = s.misc[0];
  const int nbeg = (int)((long)a.N * blockIdx.x / gridDim.x);
  const int nend = (int)((long)a.N * (blockIdx.x + 1) / gridDim.x);
  const int passes = (nend - nbeg + NPB - 1) / NPB;
  auto npts_of = [&](int i) { return min(NPB, nend - nbeg - i * NPB); };

  // ---- front warps: constants, records, psi1 and m of pass i
  auto front = [&](int i) {
    const int rt = tid - NTS, rw = rt >> 5, n0 = nbeg + i * NPB, npts = npts_of(i);
    auto slot = [&](int pt) { return PointSlot<T>(s.pd + ((i & 1) * NPB + pt) * PDN, s.rec + (size_t)((i & 1) * NPB + pt) * M * RL); };
    for (int pt = rw; pt < npts; pt += NF)
      consts_of<T, S>(a, s.ell2, s.lnl, etab, lsf, slot(pt), n0 + pt, Q, lane, &s_flag[i & 1][pt]);
    if (rw == 0 && lane >= npts && lane < NPB) s_flag[i & 1][lane] = 0;
    warps_sync<1, NF>();
    for (int t = rt; t < npts * M; t += NF * 32) {
      const int pt = t / M, ia = t - pt * M;
      const T v1 = row_of<T, QC>(s.z + ia * ZL, etab, slot(pt), Q, ia, &s_flag[i & 1][pt]);
      s.p1[pt * M + ia] = v1;
      if (a.psi1) a.psi1[(size_t)(n0 + pt) * M + ia] = Num<T>::st(v1);
    }
    warps_sync<1, NF>();
    for (int pt = rw; pt < npts; pt += NF) {   // m = psi1 . A_d, a warp a point
#pragma unroll
      for (int d = 0; d < DB; ++d) {
        if (d < D) {
          T mm = Num<T>::zero();
          for (int ia = lane; ia < M; ia += 32) mm = fma_(s.p1[pt * M + ia], s.As[d * M + ia], mm);
          mm = warp_sum(mm);
          if (lane == 0) {
            s.ms[((i % 3) * NPB + pt) * DMAX + d] = mm;
            if (a.m_out) a.m_out[(size_t)(n0 + pt) * D + d] = Num<T>::st(mm);
          }
        }
      }
    }
    warps_sync<1, NF>();
  };
  // ---- front warps: v of pass i from the sweep warps' sums, a thread an output
  auto finish = [&](int i) {
    const int rt = tid - NTS, pt = rt / DB, d = rt - pt * DB;
    if (rt < K && pt < npts_of(i) && d < D && a.v_out) {
      const T* r = s.red + (size_t)(i & 1) * NS * K + rt;
      T v = r[0];
      for (int w = 1; w < NS; ++w) v = add(v, r[w * K]);
      const T mm = s.ms[((i % 3) * NPB + pt) * DMAX + d];
      a.v_out[(size_t)(nbeg + i * NPB + pt) * D + d] = Num<T>::st(sub(add(s.misc[1], v), mul(mm, mm)));
    }
  };

  if (front_warp) {
    if (passes > 0) front(0);
  } else {
    stage_pairs<T, QC, NS, 2>(s.z, s.inv4l, Q, M, P, D, a.B, false, s.pab, s.G, s.Bs,
                              reinterpret_cast<T*>(s.G));
  }
  __syncthreads();
  for (int i = 0; i < passes; ++i) {
    if (front_warp) {
      if (i > 0) finish(i - 1);
      if (i + 1 < passes) front(i + 1);
    } else {
      const R* rec = s.rec + (size_t)(i & 1) * NPB * M * RL;
      int general = 0;
      if (X::TAB) {
#pragma unroll
        for (int pt = 0; pt < NPB; ++pt) general |= s_flag[i & 1][pt];
      }
      T vacc[K];
#pragma unroll
      for (int k = 0; k < K; ++k) vacc[k] = Num<T>::zero();
      constexpr int E = sizeof(T);
      const saddr ar = sm_addr(rec), aG = sm_addr(s.G), aB = sm_addr(s.Bs), ap = use_pab ? sm_addr(s.pab) : 0u,
                  at = sm_addr(s.tab);
      const saddr ps_ = M * (RL * E);   // from one point's records to the next
      for (int p = tid; p < P; p += NTS) {
        p = GPK_IDX(p, P, 3);
        int ia, ib;
        if (use_pab) {
          const int ab = lds_u16(ap + 2 * p);
          ia = ab >> 8;
          ib = ab & 0xff;
        } else {
          pair_of(p, ia, ib);
        }
        T w[DB];
#pragma unroll
        for (int d = 0; d < DB; ++d) w[d] = d < D ? ldsv<T>(aB + (d * P + p) * E) : Num<T>::zero();
        const R gab = ldsv<R>(aG + p * E);
        saddr ra = ar + ia * (RL * E), rb = ar + ib * (RL * E);
        if (!general) {
          // branch-free, so that the NPB points' exps interleave; in a pass with fewer points the
          // extra slots run on stale tables and their sums are never read
          R arg[NPB];
#pragma unroll
          for (int pt = 0; pt < NPB; ++pt) {
            arg[pt] = X::template arg<QC>(ra, rb, gab);
            ra += ps_;
            rb += ps_;
          }
#pragma unroll
          for (int pt = 0; pt < NPB; ++pt) {
            const T ps = X::ev(arg[pt], at);
#pragma unroll
            for (int d = 0; d < DB; ++d) acc_fma(vacc[pt * DB + d], w[d], ps);
          }
        } else {
          const int npts = npts_of(i);
#pragma unroll
          for (int pt = 0; pt < NPB; ++pt) {
            if (pt < npts) {
              const T ps = s_flag[i & 1][pt]
                               ? psi2_general(s.z + ia * ZL, s.z + ib * ZL, s.pd + ((i & 1) * NPB + pt) * PDN, s.inv4l,
                                              lsf, Q, s.tab)
                               : X::ev(X::template arg<QC>(ra, rb, gab), at);
#pragma unroll
              for (int d = 0; d < DB; ++d) acc_fma(vacc[pt * DB + d], w[d], ps);
            }
            ra += ps_;
            rb += ps_;
          }
        }
      }
      T t[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) t[k] = k < K ? acc_done(vacc[k]) : Num<T>::zero();
      warp_sum_many<8>(t);
      if ((lane & 3) == 0 && (lane >> 2) < K) s.red[((size_t)(i & 1) * NS + (tid >> 5)) * K + (lane >> 2)] = t[0];
    }
    __syncthreads();
  }
  if (front_warp && passes > 0) finish(passes - 1);
}

// ---------------------------------------------------------------------------------
// Forward with psi2 per point written out [N, M, M] (psi1 optionally): the sweep warps leave point
// i's packed pairs in shared memory as storage values while they write point i - 1's full square
// from the other buffer, each row as consecutive columns (straight from the sweep, the entries
// above the diagonal are one 8-byte store per 32-byte sector); the front warps form point i + 1.
// N = 1000, Q = 2, M = 100 (81 MB): 67 -> 45 us; FP32 24 us.  The double-float pairs become float64 by
// integer operations (exp2_fx_double): two conversions
// and an addition on the FP64 pipe took longer than the sweep itself.
template <typename T>
struct OSmem {
  typedef typename PairExp<T>::R R;
  typedef typename Num<T>::store_t S;
  float2* tab;
  T* z;      // [M][zlen]
  T* ell2;   // [QMAX]
  T* lnl;    // [QMAX]
  T* inv4l;  // [QMAX]
  T* misc;   // [4]
  T* pd;     // [2][PDN]
  R* rec;    // [2][M][rec_len]
  S* L;      // [nl][P]
  R* G;      // [P] or nullptr
  unsigned short* pab;   // [P] or nullptr
};
template <typename T>
__host__ __device__ inline size_t ocarve(OSmem<T>* out, char* base, int M, int QC, int P, int ng, int pab, int nl) {
  typedef typename PairExp<T>::R R;
  typedef typename Num<T>::store_t S;
  OSmem<T> s;
  size_t o = 0;
  auto take = [&](size_t n) {
    char* p = base + o;
    o += n;
    return p;
  };
  const size_t e = sizeof(T);
  s.tab = (float2*)take(PairExp<T>::TAB * sizeof(float2));
  s.z = (T*)take((size_t)zlen(QC) * M * e);
  s.ell2 = (T*)take(QMAX * e);
  s.lnl = (T*)take(QMAX * e);
  s.inv4l = (T*)take(QMAX * e);
  s.misc = (T*)take(4 * e);
  s.pd = (T*)take(2 * PDN * e);
  s.rec = (R*)take(2 * (size_t)M * rec_len(QC) * e);
  s.L = (S*)take((size_t)nl * P * e);
  s.G = ng ? (R*)take((size_t)ng * e) : nullptr;
  s.pab = pab ? (unsigned short*)take((size_t)P * sizeof(unsigned short)) : nullptr;
  if (out) *out = s;
  return o;
}

template <typename T, int QC, int NS, int NF>
__global__ void __launch_bounds__((NS + NF) * 32, NS < 8 ? 4 : NS < 12 ? 2 : 1)
    psi_out_kernel(PsiArgs<typename Num<T>::store_t> a, int use_pab, int nl) {
  typedef typename Num<T>::store_t S;
  typedef PairExp<T> X;
  typedef typename X::R R;
  constexpr int RL = rec_len(QC), ZL = zlen(QC), NTH = (NS + NF) * 32, NTS = NS * 32;
  extern __shared__ __align__(16) char smem_raw[];
  const int M = a.M, Q = exact_q(QC) ? QC : a.Q;
  const int P = M * (M + 1) / 2;
  OSmem<T> s;
  ocarve<T>(&s, smem_raw, M, QC, P, a.g_smem ? P : 0, use_pab, nl);
  __shared__ int s_flag[2];
  const ExpTab etab{s.tab};
  const int tid = threadIdx.x, lane = tid & 31;
  const bool front_warp = tid >= NTS;
  load_pair_table<T>(s.tab);
#pragma unroll 1
  for (int i = tid; i < M * ZL; i += NTH) {
    const int ia = i / ZL, q = i - ia * ZL;
    s.z[i] = q < Q ? Num<T>::ld(a.Z[ia * Q + q]) : Num<T>::zero();
  }
  __syncthreads();
  if (tid < Q) {
    const T lnl = Num<T>::ld(static_cast<S>(a.lls2[tid]));
    const T l2 = exp_tab(lnl, etab);
    s.lnl[tid] = lnl;
    s.ell2[tid] = l2;
    s.inv4l[tid] = recip(mul(l2, Num<T>::c(4.f)));
  }
  const T lsf = Num<T>::ld(static_cast<S>(a.lsf2[0]));
  __syncthreads();
  const int nbeg = (int)((long)a.N * blockIdx.x / gridDim.x);
  const int nend = (int)((long)a.N * (blockIdx.x + 1) / gridDim.x);
  const int cnt = nend - nbeg;
  auto front = [&](int i) {
    const int rt = tid - NTS, n = nbeg + i;
    const PointSlot<T> ps(s.pd + (i & 1) * PDN, s.rec + (size_t)(i & 1) * M * RL);
    if (rt < 32) consts_of<T, S>(a, s.ell2, s.lnl, etab, lsf, ps, n, Q, lane, &s_flag[i & 1]);
    warps_sync<1, NF>();
    for (int ia = rt; ia < M; ia += NF * 32) {
      const T v1 = row_of<T, QC>(s.z + ia * ZL, etab, ps, Q, ia, &s_flag[i & 1]);
      if (a.psi1) a.psi1[(size_t)n * M + ia] = Num<T>::st(v1);
    }
  };
  if (front_warp) {
    if (cnt > 0) front(0);
  } else {
    stage_pairs<T, QC, NS, 2>(s.z, s.inv4l, Q, M, P, 0, (const S*)nullptr, false, s.pab, s.G, (T*)nullptr,
                              (T*)nullptr);
  }
  __syncthreads();
  for (int i = 0; i <= cnt; ++i) {
    if (front_warp) {
      if (i + 1 < cnt) front(i + 1);
    } else {
      if (i < cnt) {
        S* L = s.L + (size_t)(i & (nl - 1)) * P;
        const R* rec = s.rec + (size_t)(i & 1) * M * RL;
        const bool general = X::TAB && s_flag[i & 1];
        constexpr int E = sizeof(T);
        const saddr ar = sm_addr(rec), aG = a.g_smem ? sm_addr(s.G) : 0u, aL = sm_addr(L),
                    ap = use_pab ? sm_addr(s.pab) : 0u, at = sm_addr(s.tab);
        // two pairs (p, p + NTS) per iteration, so that their chains interleave
        for (int p0 = tid; p0 < P; p0 += 2 * NTS) {
          R arg[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int p = u && p0 + NTS < P ? p0 + NTS : p0;
            int ia, ib;
            if (use_pab) {
              const int ab = lds_u16(ap + 2 * p);
              ia = ab >> 8;
              ib = ab & 0xff;
            } else {
              pair_of(p, ia, ib);
            }
            if (general) {
              sts(aL + p * E, Num<T>::st(psi2_general(s.z + ia * ZL, s.z + ib * ZL, s.pd + (i & 1) * PDN, s.inv4l, lsf, Q,
                                                      s.tab)));
            } else {
              arg[u] = X::template arg<QC>(ar + ia * (RL * E), ar + ib * (RL * E),
                                           a.g_smem ? ldsv<R>(aG + p * E)
                                                    : pair_G<T, QC>(s.z + ia * ZL, s.z + ib * ZL, s.inv4l, Q));
            }
          }
          if (!general) {
#pragma unroll
            for (int u = 0; u < 2; ++u) sts(aL + (u && p0 + NTS < P ? p0 + NTS : p0) * E, X::ev_st(arg[u], at));
          }
        }
      }
      if (nl == 1) warps_sync<2, NS>();
      const int w = nl == 1 ? i : i - 1;   // the point whose square goes out, a warp a row, 128 columns at a time
      if (w >= 0 && w < cnt) {
        constexpr int E = sizeof(T);
        const saddr aL = sm_addr(s.L + (size_t)(w & (nl - 1)) * P);
        S* const out = a.psi2 + (size_t)(nbeg + w) * M * M;
        for (int c0 = 0; c0 < M; c0 += 128) {
          saddr up[4];   // the lane's columns: where their entries below the diagonal begin
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int b = c0 + lane + 32 * k;
            up[k] = aL + b * (b + 1) / 2 * E;
          }
          for (int ia = tid >> 5; ia < M; ia += NS) {
            const saddr row = aL + (ia * (ia + 1) / 2 + c0 + lane) * E;
            S* const o = out + (size_t)ia * M + c0 + lane;
            const int left = M - c0 - lane, below = ia - c0 - lane;   // columns left, columns up to the diagonal
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (32 * k < left) {
                S v;
                lds_st(32 * k <= below ? row + 32 * k * E : up[k] + ia * E, v);
                o[32 * k] = v;
              }
            }
          }
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------
// Rollout in double-float precision: one CTA, T dependent steps, each taking the previous step's
// moments, so a step's latency is the cost.  Against the general kernel's step (four barriers,
// logarithms and divisions in sequence, two double-float butterflies; 5.2 us at M = 50, Q = 2):
//  * the normalisers enter as products of reciprocal square roots (no logarithm, no division), the
//    point-dependent scale of psi2 multiplying the finished sum;
//  * every thread that needs the step's constants forms them itself from the summed partials (no
//    exchange), so a step has two barriers: records ready, partial sums ready.  CH_REC warps form
//    the records (128 rows at a time; those without rows sit out), CH_PSI1 warps psi1 and its sums
//    beside them, CH_SWEEP warps the pairs;
//  * the sums over threads are integer sums, in units of 2^-57 of a warp's largest lane, so that a state far
//    from every pseudo-input keeps its bits (psi1 beside the warp's nearest pseudo-input's): three 32-bit
//    warp reductions a sum, and one for the scale, for what took five shuffle-and-add levels.  In units of
//    2^-60 of sum |A| and sum |B| instead, a mean 2^-40 of sum |A| had 20 bits left (2.47 us a step at M = 50,
//    Q = 2, 2.56 now; the warps' sums brought to one scale by each thread instead of a lane each 2.8);
//  * with up to four pairs a thread, their G and B stay in registers.
// Measured per step: M = 50, Q = 2: 5.2 -> 2.6 us; M = 100: 9.2 -> 4.6; M = 30, Q = 3: 6.0 -> 5.2;
// M = 10, Q = 1: 3.8 -> 2.4 (the dependent chain alone).  At M = 50 the issue rate of one SM bounds the
// pair phase (~5000 instructions a step): twelve sweep warps of four pairs a
// thread take fewer of them than twenty of two (each warp pays ~100 for its reduction).
constexpr int CH_REC = 4, CH_PSI1 = 4, CH_SWEEP = 12, CH_KP = 4;
constexpr int CH_NTH = (CH_REC + CH_PSI1 + CH_SWEEP) * 32;
// v 2^F as an integer (|v 2^F| < 2^57)
__device__ __forceinline__ long long fx_dyn(float x, int F) {
  const unsigned b = __float_as_uint(x);
  const int s = max(0, min(189 - F - (int)((b >> 23) & 0xffu), 63));
  const long long v = (long long)(((unsigned long long)(((b & 0x7fffffu) | 0x800000u) << 7) << 32) >> s);
  return (int)b < 0 ? -v : v;
}
// the warp's sum of |x| < 2^57 (32 lanes stay below 2^62)
__device__ __forceinline__ long long warp_sum_fx(long long x) {
  const unsigned l0 = (unsigned)x & 0x3ffffffu, l1 = (unsigned)(x >> 26) & 0x3ffffffu;
  const int l2 = (int)(x >> 52);
  const unsigned s0 = __reduce_add_sync(0xffffffffu, l0), s1 = __reduce_add_sync(0xffffffffu, l1);
  const int s2 = __reduce_add_sync(0xffffffffu, l2);
  return (long long)s0 + ((long long)s1 << 26) + ((long long)s2 << 52);
}
// an integer as a double-float in units of 2^16
__device__ __forceinline__ df64 df_of_fx(long long x) {
  const float h = (float)(int)(x >> 38), m = (float)(int)((x >> 16) & 0x3fffff), l = (float)(int)(x & 0xffff);
  // 26, 22 and 16 bits; h may round (its error is recovered exactly)
  const int he = (int)(x >> 38) - __float2int_rn(h);
  const df64 a = two_sum(__fmul_rn(h, 4194304.f), __fmaf_rn((float)he, 4194304.f, m));
  return add(a, __fmul_rn(l, 1.52587890625e-05f));
}
// the warp's sum of one value a lane, times 2^-off: an integer in units of 2^(e - 183 - off), e the largest
// lane's exponent field, with e - off + 128 in its last nine bits (2^-48 of that lane); 511: not finite
__device__ __forceinline__ long long warp_sum_scaled(df64 v, int off) {
  const int e = __reduce_max_sync(0xffffffffu, (int)((__float_as_uint(v.hi) >> 23) & 0xffu));
  const long long s = warp_sum_fx(fx_dyn(v.hi, 183 - e) + fx_dyn(v.lo, 183 - e));
  return ((s + 256) & ~511LL) | (e == 255 ? 511 : e - off + 128);
}
// the lanes' such sums x (0: none), G bits that their number needs: the total, a double-float times 2^e (e >= -240:
// less is zero in any case)
template <int G>
__device__ __forceinline__ df64 sum_of_scaled(long long x, int& e) {
  const int code = (int)x & 511, top = __reduce_max_sync(0xffffffffu, code);
  const long long s = warp_sum_fx(x >> min(top - code + G, 63));
  e = max(top + G - 295, -240);
  df64 r = df_of_fx(s);
  r.hi = top == 511 ? __int_as_float(0x7fffffff) : r.hi;
  return r;
}
// a 2^e, -252 <= e <= 254, without a branch
__device__ __forceinline__ df64 scale2_by(df64 a, int e) {
  const float p = pow2f(e >> 1), q = pow2f(e - (e >> 1));
  return make_df(a.hi * p * q, a.lo * p * q);
}
struct ChSmem {
  float2* tab;
  df64 *z, *As, *ell2, *sl, *inv4l, *misc;   // misc: sf2, then a step's normalisers of psi1 and psi2
  long long* rec;    // [M][rec_len]
  long long* part;   // [QC][CH_PSI1] sums of m, then [QC][CH_SWEEP] of v (warp_sum_scaled)
  long long* G;      // [P]
  df64* Bs;          // [QC * P]
  unsigned short* pab;   // [P]
};
__host__ __device__ inline size_t chcarve(ChSmem* out, char* base, int M, int QC, int P) {
  ChSmem s;
  size_t o = 0;
  auto take = [&](size_t n) {
    char* p = base + o;
    o += n;
    return p;
  };
  s.tab = (float2*)take(kFxTab * sizeof(float2));
  s.z = (df64*)take((size_t)zlen(QC) * M * 8);
  s.As = (df64*)take((size_t)QC * M * 8);
  s.ell2 = (df64*)take(QC * 8);
  s.sl = (df64*)take(QC * 8);
  s.inv4l = (df64*)take(QMAX * 8);
  s.misc = (df64*)take(4 * 8);
  s.part = (long long*)take((size_t)QC * (CH_PSI1 + CH_SWEEP) * 8);   // (16-byte aligned: read in pairs)
  s.rec = (long long*)take((size_t)M * rec_len(QC) * 8);
  s.G = (long long*)take((size_t)P * 8);
  s.Bs = (df64*)take((size_t)QC * P * 8);
  s.pab = (unsigned short*)take((size_t)P * 2);
  if (out) *out = s;
  return o;
}

// a sweep thread's pairs of a step outside the fixed-point range (rare, so out of line): the
// exponents in double-float, psi2 without its point-dependent scale
template <int QC>
struct ChSums {
  df64 v[QC];
};
template <int QC>
__device__ __noinline__ ChSums<QC> chain_general(const double* mu, const double* var, const df64* z, const df64* ell2,
                                                 const df64* inv4l, const float2* tab, const unsigned short* pab,
                                                 const df64* Bs, int Q, int p0, int np, int P) {
  df64 m[QC], c[QC];
  ChSums<QC> r;
#pragma unroll
  for (int q = 0; q < QC; ++q) {
    const df64 v = df_from_double(q < Q ? var[q] : 0.0);
    m[q] = df_from_double(q < Q ? mu[q] : 0.0);
    c[q] = recip(add(ell2[q], add(v, v)));
    r.v[q] = make_df(0.f);
  }
  for (int p = p0; p < P; p += np) {
    const int ia = pab[p] >> 8, ib = pab[p] & 0xff;
    df64 x = make_df(0.f);
#pragma unroll
    for (int q = 0; q < QC; ++q) {
      const df64 za = z[ia * zlen(QC) + q], zb = z[ib * zlen(QC) + q];
      const df64 u = sub(m[q], scale2(add(za, zb), -1)), d = sub(za, zb);
      x = sub(x, add(mul(mul(u, u), c[q]), mul(mul(d, d), inv4l[q])));
    }
    const df64 ps = exp_pair(x, ExpTab{tab});
#pragma unroll
    for (int d = 0; d < QC; ++d) acc_fma(r.v[d], Bs[d * P + p], ps);
  }
  return r;
}

template <int QC, bool REGS>
__global__ void __launch_bounds__(CH_NTH, 1) psi_chain_kernel(PsiArgs<double> a) {
  typedef PairExp<df64> X;
  constexpr int RL = rec_len(QC), ZL = zlen(QC), NTH = CH_NTH, NTS = CH_SWEEP * 32, KP = CH_KP;
  extern __shared__ __align__(16) char smem_raw[];
  const int M = a.M, Q = a.Q, P = M * (M + 1) / 2, T = a.N;
  ChSmem s;
  chcarve(&s, smem_raw, M, QC, P);
  __shared__ int s_flag[2];
  const ExpTab etab{s.tab};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool sweep_warp = warp >= CH_REC + CH_PSI1, rec_warp = warp < CH_REC;
  load_exp2_table(s.tab);
#pragma unroll 1
  for (int i = tid; i < M * ZL; i += NTH) {
    const int ia = i / ZL, q = i - ia * ZL;
    s.z[i] = q < Q ? df_from_double(a.Z[ia * Q + q]) : make_df(0.f);
  }
  if (tid < 2) s_flag[tid] = 0;
  for (int i = tid; i < QC * (CH_PSI1 + CH_SWEEP); i += NTH) s.part[i] = 0;
  __syncthreads();
  if (tid < QC) {
    const df64 l2 = tid < Q ? exp_tab(df_from_double(a.lls2[tid]), etab) : make_df(1.f);
    s.ell2[tid] = l2;
    s.sl[tid] = sqrt_(l2);
    s.inv4l[tid] = recip(mul(l2, make_df(4.f)));
  }
  if (tid == 32) s.misc[0] = exp_tab(df_from_double(a.lsf2[0]), etab);
#pragma unroll 1
  for (int i = tid; i < QC * M; i += NTH) {
    const int d = i / M;
    s.As[i] = d < Q ? df_from_double(a.A[i]) : make_df(0.f);
  }
  __syncthreads();
#pragma unroll 1
  for (int p = tid; p < P; p += NTH) {
    int ia, ib;
    pair_of(p, ia, ib);
    s.pab[p] = (unsigned short)((ia << 8) | ib);
    s.G[p] = pair_G<df64, QC>(s.z + ia * ZL, s.z + ib * ZL, s.inv4l, Q);
    for (int d = 0; d < QC; ++d) {
      df64 w = make_df(0.f);
      if (d < Q) {
        const double* B = a.B + (size_t)d * M * M;
        w = df_from_double(B[ia * M + ib]);
        if (ia != ib) w = add(w, df_from_double(B[ib * M + ia]));
      }
      s.Bs[d * P + p] = w;
    }
  }
  __syncthreads();
  const df64 sf2 = s.misc[0], kq = make_df(8.493217826e-01f, 1.769906000e-08f);   // sqrt(log2(e) / 2)
  // the pairs of a sweep thread, their G and B
  const int st = tid - (CH_REC + CH_PSI1) * 32;
  long long g[KP];
  df64 w[KP][QC];
  int off[KP];
  if (REGS && sweep_warp) {
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int p = st + k * NTS;
      const bool in = p < P;
      g[k] = in ? s.G[p] : 0;
      off[k] = in ? s.pab[p] : 0;
#pragma unroll
      for (int d = 0; d < QC; ++d) w[k][d] = in ? s.Bs[d * P + p] : make_df(0.f);
    }
  }
  __syncthreads();
  for (int t = 0; t <= T; ++t) {
    if (!sweep_warp) {
      // rows of this thread: from r0 in steps of 128 (a warp without rows only keeps the barriers)
      const int r0 = rec_warp ? tid : tid - CH_REC * 32;
      const bool live_warp = (r0 & ~31) < M;
      df64 m[QC], v[QC];
#pragma unroll
      for (int d = 0; d < QC; ++d) m[d] = v[d] = make_df(0.f);
      if (live_warp) {
        if (t == 0) {
#pragma unroll
          for (int d = 0; d < QC; ++d)
            if (d < Q) m[d] = df_from_double(a.mu[d]), v[d] = df_from_double(a.var[d]);
        } else {
          // ---- the previous step's moments from the partial sums (each warp for itself)
          const df64 K1 = s.misc[1], F2 = s.misc[2];
          df64 mu[QC];   // m times 2^64 where it is below ~2^-96 (its low word would leave the float range)
          int up[QC];
#pragma unroll
          for (int d = 0; d < QC; ++d) {
            int em, ev;
            const df64 rm = sum_of_scaled<2>(lane < CH_PSI1 ? s.part[d * CH_PSI1 + lane] : 0, em);
            const df64 rv = sum_of_scaled<4>(lane < CH_SWEEP ? s.part[QC * CH_PSI1 + d * CH_SWEEP + lane] : 0, ev);
            up[d] = em < -142 ? 64 : 0;
            mu[d] = mul(K1, scale2_by(rm, em + up[d]));
            const float down = pow2f(-up[d]);
            m[d] = make_df(mu[d].hi * down, mu[d].lo * down);
            v[d] = sub(fma_(F2, scale2_by(rv, ev), sf2), mul(m[d], m[d]));
          }
          if (tid == 0) {   // (before the barrier: the general form reads them)
#pragma unroll
            for (int d = 0; d < QC; ++d)
              if (d < Q) {
                const double md = df_to_double_int(mu[d]);
                a.m_out[(size_t)(t - 1) * Q + d] = up[d] ? md * 5.42101086242752217e-20 : md;   // 2^-64
                a.v_out[(size_t)(t - 1) * Q + d] = df_to_double_int(v[d]);
              }
          }
        }
      }
      if (t == T) break;
      if (rec_warp) {
        df64 r2[QC];
        if (live_warp) {
          // ---- this thread's records
          bool minus = false;
#pragma unroll
          for (int q = 0; q < QC; ++q) {
            const df64 l = s.ell2[q];
            r2[q] = rsqrt_(add(l, add(v[q], v[q])));
            minus |= !(v[q].hi >= -1e-6f * l.hi);   // (also NaN)
          }
          for (int ia = r0; ia < M; ia += CH_REC * 32) {
            df64 s2 = make_df(0.f), tq[QC];
#pragma unroll
            for (int q = 0; q < QC; ++q) {
              tq[q] = mul(sub(m[q], s.z[ia * ZL + q]), mul(r2[q], kq));
              s2 = fma_(tq[q], tq[q], s2);
            }
            const bool in = s2.hi < 1e38f && !minus;
            if (!in) s_flag[t & 1] = 1;
            const bool live = in && s2.hi <= 127.5f;
            long long* r = s.rec + ia * RL;
            r[0] = live ? X::u_of(scale2(neg(s2), -1)) : X::dead_u();
#pragma unroll
            for (int q = 0; q < QC; ++q) r[1 + q] = live ? X::t_of(tq[q]) : X::t_of(make_df(0.f));
          }
        }
        __syncthreads();   // records ready
        if (warp == 0) {
          df64 F2 = mul(sf2, sf2);
#pragma unroll
          for (int q = 0; q < QC; ++q)
            if (q < Q) F2 = mul(F2, mul(s.sl[q], r2[q]));
          if (lane == 0) {
            s.misc[2] = F2;
            s_flag[(t + 1) & 1] = 0;
          }
        }
      } else {
        // ---- psi1 and its sums
        df64 mm[QC], r1[QC], K1 = sf2;
        int off = 0;   // the terms are 2^off psi1 / K1, 2^-off that of the warp's nearest row
        if (live_warp) {
          const bool one_each = M <= CH_PSI1 * 32;   // (the tables of more rows do not fit beside two inputs)
          const unsigned row_lanes = 0xffffffffu >> max(32 - (M - (r0 & ~31)), 0);
#pragma unroll
          for (int q = 0; q < QC; ++q) {
            mm[q] = make_df(0.f);
            r1[q] = rsqrt_(add(s.ell2[q], v[q]));
            if (q < Q) K1 = mul(K1, mul(s.sl[q], r1[q]));
            r1[q] = mul(r1[q], kq);
          }
          for (int ia = r0; ia < M; ia += CH_PSI1 * 32) {
            df64 e = make_df(0.f);
#pragma unroll
            for (int q = 0; q < QC; ++q) {
              const df64 x = mul(sub(m[q], s.z[ia * ZL + q]), r1[q]);
              e = fma_(x, x, e);
            }
            // psi1 / K1 = 2^-e
            if (one_each) off = (int)__reduce_min_sync(row_lanes, (unsigned)fminf(fmaxf(e.hi, 0.f), 120.f));
            const float left = e.hi - (float)off;
            const df64 p1 = left < 126.f ? exp2_fx(fx52_of(neg(e)) + kFxHalf + ((long long)off << 52), sm_addr(s.tab))
                                         : (left >= 126.f ? make_df(0.f) : make_df(__int_as_float(0x7fffffff)));
#pragma unroll
            for (int d = 0; d < QC; ++d) acc_fma(mm[d], p1, s.As[d * M + ia]);
          }
        }
        __syncthreads();
        if (live_warp) {
#pragma unroll
          for (int d = 0; d < QC; ++d) {
            const long long x = warp_sum_scaled(acc_done(mm[d]), off);
            if (lane == 0) s.part[d * CH_PSI1 + warp - CH_REC] = x;
          }
          if (warp == CH_REC && lane == 0) s.misc[1] = K1;
        }
      }
      __syncthreads();   // partial sums ready
    } else {
      if (t == T) break;
      __syncthreads();
      const bool general = s_flag[t & 1] != 0;
      const saddr ar = sm_addr(s.rec), at = sm_addr(s.tab);
      df64 vv[QC];
#pragma unroll
      for (int d = 0; d < QC; ++d) vv[d] = make_df(0.f);
      if (!general) {
        if (REGS) {
          long long arg[KP];
#pragma unroll
          for (int k = 0; k < KP; ++k)
            arg[k] = X::template arg<QC>(ar + (off[k] >> 8) * (RL * 8), ar + (off[k] & 0xff) * (RL * 8), g[k]);
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            const df64 ps = X::ev(arg[k], at);
#pragma unroll
            for (int d = 0; d < QC; ++d) acc_fma(vv[d], w[k][d], ps);
          }
        } else {
          for (int p = st; p < P; p += NTS) {
            const int ab = s.pab[p];
            const df64 ps = X::ev(X::template arg<QC>(ar + (ab >> 8) * (RL * 8), ar + (ab & 0xff) * (RL * 8), s.G[p]), at);
#pragma unroll
            for (int d = 0; d < QC; ++d) acc_fma(vv[d], s.Bs[d * P + p], ps);
          }
        }
      } else {
        // outside the fixed-point range: from the moments as they were written out
        const ChSums<QC> r = chain_general<QC>(t ? a.m_out + (size_t)(t - 1) * Q : a.mu,
                                               t ? a.v_out + (size_t)(t - 1) * Q : a.var, s.z, s.ell2, s.inv4l, s.tab,
                                               s.pab, s.Bs, Q, st, NTS, P);
#pragma unroll
        for (int d = 0; d < QC; ++d) vv[d] = r.v[d];
      }
#pragma unroll
      for (int d = 0; d < QC; ++d) {
        const long long x = warp_sum_scaled(acc_done(vv[d]), 0);
        if (lane == 0) s.part[QC * CH_PSI1 + d * CH_SWEEP + warp - CH_REC - CH_PSI1] = x;
      }
      __syncthreads();
    }
  }
}

template <typename T, int NPB, int PPT, int QC, int DB>
int run_fwd_gen(const PsiArgs<typename Num<T>::store_t>& a_in, cudaStream_t st) {
  PsiArgs<typename Num<T>::store_t> a = a_in;
  const int P = a.M * (a.M + 1) / 2;
  const bool contract = a.A && a.B && (a.m_out || a.v_out);
  const int D = contract ? a.Dout : 0, nbs = D * P;
  // G and the symmetrised B in shared memory as far as they fit; B first (from global memory it
  // costs two loads and conversions per pair, G a few operations per dimension)
  auto bytes = [&](int ng, int nb) { return fwd_smem_bytes(a.M, a.Q, QC, D, NPB, sizeof(T), ng, nb); };
  a.bs_smem = contract && bytes(0, nbs) <= SMEM_CAP;
  a.g_smem = bytes(P, a.bs_smem ? nbs : 0) <= SMEM_CAP;
  const size_t sm = bytes(a.g_smem ? P : 0, a.bs_smem ? nbs : 0);
  auto k = psi_fwd_gen_kernel<T, NPB, PPT, QC, DB>;
  gpk::allow_smem(k, sm, SMEM_STATIC);
  int resident = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k, NT, sm);
  resident = resident < 1 ? 1 : (resident > 2 ? 2 : resident);
  int grid = a.chain ? 1 : gpk::sm_count() * resident;   // a rollout is one CTA's sequence
  if (grid > a.N) grid = a.N;
  if (grid < 1) return GPK_OK;
  k<<<grid, NT, sm, st>>>(a);
  return gpk::check_launch("psi_fwd");
}

// the double-float rollout kernel, or -1 where its tables do not fit
template <int QC>
int run_chain(const PsiArgs<double>& a, cudaStream_t st) {
  const int P = a.M * (a.M + 1) / 2;
  const size_t sm = chcarve(nullptr, nullptr, a.M, QC, P);
  if (sm > SMEM_CAP || a.M > 255) return -1;
  if (a.N < 1) return GPK_OK;
  auto k = P <= CH_KP * CH_SWEEP * 32 ? psi_chain_kernel<QC, true> : psi_chain_kernel<QC, false>;
  gpk::allow_smem(k, sm, SMEM_STATIC);
  k<<<1, CH_NTH, sm, st>>>(a);
  return gpk::check_launch("psi_rollout");
}
template <int QC>
int run_chain(const PsiArgs<float>&, cudaStream_t) { return -1; }

// points per pass: 4 for Dout <= 2, 2 for Dout <= 4 (so 2*NPB*Dout sums fit one reduction)
template <typename T, int QC>
int fwd_gen(const PsiArgs<typename Num<T>::store_t>& a, bool sum, bool contract, int P, cudaStream_t st) {
  if (sum) {
    if (P <= 4 * NT) return run_fwd_gen<T, 2, 4, QC, 4>(a, st);
    return run_fwd_gen<T, 2, 16, QC, 4>(a, st);
  }
  if (a.chain) {   // one point per pass: each point needs the previous one's moments
    const int rc = run_chain<QC == 2 ? 2 : 4>(a, st);
    if (rc != -1) return rc;
    if (a.Dout == 1) return run_fwd_gen<T, 1, 0, QC, 1>(a, st);
    if (a.Dout == 2) return run_fwd_gen<T, 1, 0, QC, 2>(a, st);
    return run_fwd_gen<T, 1, 0, QC, 4>(a, st);
  }
  if (contract && a.Dout == 1 && !a.psi2) {
    // points per pass: a pass evaluates all its slots at ~75 instructions each beside ~100 a pair for
    // its constants, so that with few points a CTA a width that divides them leaves fewer slots idle
    // (M = 200, Q = 2, with B read along its rows: 100 points 80 -> 55 us, 777 points 138 -> 119)
    const int per = gpk::ceil_div(a.N, gpk::sm_count());
    int best = 4;
    for (int npb = 3; npb >= 1; --npb)
      if ((long)gpk::ceil_div(per, npb) * (100 + 75 * npb) < (long)gpk::ceil_div(per, best) * (100 + 75 * best)) best = npb;
    if (best == 1) return run_fwd_gen<T, 1, 0, QC, 1>(a, st);
    if (best == 2) return run_fwd_gen<T, 2, 0, QC, 1>(a, st);
    if (best == 3) return run_fwd_gen<T, 3, 0, QC, 1>(a, st);
  }
  if (!contract || a.Dout == 1) return run_fwd_gen<T, 4, 0, QC, 1>(a, st);
  if (a.Dout == 2) return run_fwd_gen<T, 4, 0, QC, 2>(a, st);
  return run_fwd_gen<T, 2, 0, QC, 4>(a, st);
}

// the moments kernel, or -1 where its tables do not fit
template <typename T, int NPB, int QC, int DB, int NS, int NF>
int run_fwd(const PsiArgs<typename Num<T>::store_t>& a, size_t cap, cudaStream_t st) {
  const int P = a.M * (a.M + 1) / 2;
  int pab = a.M <= 255;
  // whether this split is taken depends on the sizes of the full pass only, not on N
  constexpr int NPBF = DB <= 2 ? 4 : 2;
  if (mcarve<T>(nullptr, nullptr, a.M, QC, P, a.Dout, NPBF, NS, DB, pab) > cap && NS >= 16) pab = 0;
  if (mcarve<T>(nullptr, nullptr, a.M, QC, P, a.Dout, NPBF, NS, DB, pab) > cap) return -1;
  const size_t sm = mcarve<T>(nullptr, nullptr, a.M, QC, P, a.Dout, NPB, NS, DB, pab);
  auto k = psi_fwd_kernel<T, NPB, QC, DB, NS, NF>;
  gpk::allow_smem(k, sm, SMEM_STATIC);
  int grid = gpk::sm_count() * (NS < 16 ? 2 : 1);
  if (grid > a.N) grid = a.N;
  if (grid < 1) return GPK_OK;
  k<<<grid, (NS + NF) * 32, sm, st>>>(a, pab);
  return gpk::check_launch("psi_fwd");
}

template <typename T, int QC, int NS, int NF>
int fwd_npb(const PsiArgs<typename Num<T>::store_t>& a, size_t cap, cudaStream_t st) {
  // points per pass: one where every CTA has a single point (a pass evaluates all its slots), else
  // four (two for Dout > 2: eight sums a thread)
  const bool one = a.N <= gpk::sm_count() * (NS < 16 ? 2 : 1);
  if (a.Dout == 1) return one ? run_fwd<T, 1, QC, 1, NS, NF>(a, cap, st) : run_fwd<T, 4, QC, 1, NS, NF>(a, cap, st);
  if (a.Dout == 2) return one ? run_fwd<T, 1, QC, 2, NS, NF>(a, cap, st) : run_fwd<T, 4, QC, 2, NS, NF>(a, cap, st);
  return run_fwd<T, 2, QC, 4, NS, NF>(a, cap, st);
}

template <typename T, int QC, int NS, int NF>
int run_out(const PsiArgs<typename Num<T>::store_t>& a_in, size_t cap, cudaStream_t st) {
  PsiArgs<typename Num<T>::store_t> a = a_in;
  const int P = a.M * (a.M + 1) / 2;
  // G, a second buffer of pairs and the pair table as far as they fit (several CTAs an SM only with
  // all of them); G in place of the second buffer: at M = 128, Q = 8 the pairs' G from the pseudo-inputs
  // cost 226 us (N = 1000) against 113 us for a write that waits for its sweep
  const int per_sm = NS >= 12 ? 1 : NS >= 8 ? 2 : 4;
  for (int o = 0; o < (NS < 12 ? 1 : 5); ++o) {
    const int pab = (o == 0 || o == 2) && a.M <= 255, nl = o == 2 || o == 3 ? 1 : 2;
    a.g_smem = o < 4;
    const size_t sm = ocarve<T>(nullptr, nullptr, a.M, QC, P, a.g_smem ? P : 0, pab, nl);
    if (sm > cap) continue;
    auto k = psi_out_kernel<T, QC, NS, NF>;
    gpk::allow_smem(k, sm, SMEM_STATIC);
    int grid = gpk::sm_count() * per_sm;
    if (grid > a.N) grid = a.N;
    if (grid < 1) return GPK_OK;
    k<<<grid, (NS + NF) * 32, sm, st>>>(a, pab, nl);
    return gpk::check_launch("psi_out");
  }
  return -1;
}

// one input width's kernels (each width is a translation unit of its own)
template <typename T, int QC>
int launch_fwd_q(const PsiArgs<typename Num<T>::store_t>& a, cudaStream_t st) {
  const int P = a.M * (a.M + 1) / 2;
  const bool contract = a.A && a.B && (a.m_out || a.v_out);
  const bool sum = a.psi2_sum != nullptr;
  const size_t half = (SMEM_CAP - 2048) / 2;   // two CTAs an SM
  int rc = -1;
  if (!sum && !a.chain && !a.psi2 && contract) {
    // the split of the sums may not depend on N: a point's moments are the same, bit for bit, in any
    // batch (the points per pass do not enter a point's sums)
    rc = fwd_npb<T, QC, 8, 4>(a, half, st);
    if (rc == -1) rc = fwd_npb<T, QC, 16, 4>(a, SMEM_CAP, st);
  } else if (!sum && !a.chain && a.psi2 && !contract) {
    if (a.N > gpk::sm_count()) {
      rc = run_out<T, QC, 4, 2>(a, (SMEM_CAP - 4096) / 4, st);
      if (rc == -1) rc = run_out<T, QC, 8, 4>(a, half, st);
    }
    if (rc == -1) rc = run_out<T, QC, 16, 4>(a, SMEM_CAP, st);
  }
  if (rc != -1) return rc;
  if constexpr (plain_q(QC)) {
    return GPK_EUNSUPPORTED;   // the caller falls back to the catch-all width
  } else {
    return fwd_gen<T, QC>(a, sum, contract, P, st);
  }
}

// the size limits, the same for every form
template <typename S>
int check_fwd(const PsiArgs<S>& a) {
  const int P = a.M * (a.M + 1) / 2;
  const bool contract = a.A && a.B && (a.m_out || a.v_out);
  const bool sum = a.psi2_sum != nullptr;
  const int npb = a.chain ? 1 : ((sum || (contract && a.Dout > 2)) ? 2 : 4);
  const int D = contract ? a.Dout : 0;
  // accepted sizes: a pair table and the points' tables within shared memory
  const size_t need = 2048 + ((size_t)a.M * a.Q + 28 + (size_t)npb * 40 + (size_t)npb * a.M * (2 + a.Q) +
                              (size_t)D * a.M + P + 1536) * sizeof(S);
  if (need > 227 * 1024) return gpk::fail(GPK_EUNSUPPORTED, "psi_fwd: M=%d needs %zu B of shared memory", a.M, need);
  if (sum && P > PPT_MAX * NT)
    return gpk::fail(GPK_EUNSUPPORTED, "psi_fwd: psi2_sum needs M(M+1)/2 <= %d (M=%d)", PPT_MAX * NT, a.M);
  return GPK_OK;
}

// the destinations of the backward's partial block (layout in PsiArgs::part)
template <typename S>
gpk::RedPlan bwd_plan(const PsiArgs<S>& a) {
  const int M = a.M, Q = a.Q, D = a.Dout, P = M * (M + 1) / 2;
  gpk::RedPlan r{};
  r.add(a.dB, D * P, 1, M);
  r.add(a.dpsi1 ? nullptr : a.dA, D * M);
  r.add(a.dZ, M * Q);
  r.add(a.dsf2, 1);
  r.add(a.dl, Q);
  return r;
}

template <typename T, int DB, int QC, int NS, int NB, int NF>
int run_bwd(const PsiArgs<typename Num<T>::store_t>& a, const BLayout& lo, size_t sm, cudaStream_t st) {
  auto k = psi_bwd_kernel<T, DB, QC, NS, NB, NF>;
  gpk::allow_smem(k, sm, SMEM_STATIC);
  int grid = gpk::sm_count() * (NS < 12 ? 2 : 1);
  if (grid > a.N) grid = a.N;
  if (grid < 1) return GPK_OK;
  k<<<grid, (NS + NB + NF) * 32, sm, st>>>(a, lo);
  int rc = gpk::check_launch("psi_bwd");
  if (rc != GPK_OK || !a.part) return rc;
  return gpk::reduce_partials(a.part, grid, bwd_plan(a), st);
}

template <typename T, int QC, int NS, int NB, int NF>
int bwd_db(const PsiArgs<typename Num<T>::store_t>& a, const BLayout& lo, size_t sm, cudaStream_t st) {
  if (a.Dout == 1) return run_bwd<T, 1, QC, NS, NB, NF>(a, lo, sm, st);
  if (a.Dout == 2) return run_bwd<T, 2, QC, NS, NB, NF>(a, lo, sm, st);
  return run_bwd<T, 4, QC, NS, NB, NF>(a, lo, sm, st);
}

// the warp split: 12 + 4 + 4 with one CTA an SM (128 rows at a time), 6 + 2 + 2 with two
template <typename T, int QC>
int bwd_width(const PsiArgs<typename Num<T>::store_t>& a, const BLayout& lo, size_t sm, bool two, cudaStream_t st) {
  return two ? bwd_db<T, QC, 6, 2, 2>(a, lo, sm, st) : bwd_db<T, QC, 12, 4, 4>(a, lo, sm, st);
}
// widths 4 and QMAX (a translation unit of their own)
template <typename S>
using BwdWide = int (*)(const PsiArgs<S>& a, int QC, const BLayout& lo, size_t sm, bool two, cudaStream_t st);
template <typename T>
int bwd_wide(const PsiArgs<typename Num<T>::store_t>& a, int QC, const BLayout& lo, size_t sm, bool two,
             cudaStream_t st) {
  return QC == 4 ? bwd_width<T, 4>(a, lo, sm, two, st) : bwd_width<T, QMAX>(a, lo, sm, two, st);
}

template <typename T>
int launch_bwd(const PsiArgs<typename Num<T>::store_t>& a, BwdWide<typename Num<T>::store_t> wide, cudaStream_t st) {
  const int M = a.M, P = M * (M + 1) / 2;
  if (M > 512) return gpk::fail(GPK_EUNSUPPORTED, "psi_bwd: M=%d > %d", M, 512);
  const size_t cap = SMEM_CAP;
  // accepted sizes: two pair tables and the point's tables within shared memory
  const size_t need = 2048 + ((size_t)M * a.Q + 84 + (size_t)M * (1 + a.Q) + 2 * (size_t)P + (size_t)M * 9 +
                              (size_t)M * a.Q + 1536) * sizeof(T);
  if (need > 227 * 1024) return gpk::fail(GPK_EUNSUPPORTED, "psi_bwd: M=%d needs too much shared memory", M);
  const int QC = a.Q <= 2 ? 2 : a.Q <= 4 ? 4 : a.Q == 5 ? 5 : QMAX;
  auto run = [&](const BLayout& lo, size_t sm, bool two) {
    if (QC == 2) return bwd_width<T, 2>(a, lo, sm, two, st);
    if (QC == 5) return bwd_width<T, 5>(a, lo, sm, two, st);
    return wide(a, QC, lo, sm, two, st);
  };
  const int nbs = a.Dout * P, nacc = a.dB ? a.Dout * P : 0;
  auto bytes = [&](const BLayout& lo, int nb) { return bcarve<T>(nullptr, nullptr, M, QC, P, a.Dout, nb, lo); };
  auto segs = [&](int threads) { return threads / M > 8 ? 8 : (threads / M < 1 ? 1 : threads / M); };
  // two CTAs of ten warps an SM where everything fits twice (M <= ~60 in double-float precision):
  // the phases of one then overlap the other's
  {
    const BLayout lo{segs(256), P, nbs, nacc, M <= 255};
    const size_t sm = bytes(lo, 2);
    if (lo.pab && sm <= (cap - 2048) / 2) return run(lo, sm, true);
  }
  // preference: G, B, the dBhat accumulators and the pair table in shared memory; without the pair
  // table; then without G (a few operations per dimension and pair), without B (two loads and
  // conversions), without both, and without the accumulators (dBhat then accumulates in the
  // partial block, or with atomics).  Four row segments instead of five where that makes room.
  // Weights of each point's own: G stays before them (they are staged again for every point).
  const int opts[6][3] = {{P, nbs, nacc}, {a.b_stride ? P : 0, a.b_stride ? 0 : nbs, nacc},
                          {P, 0, nacc}, {0, 0, nacc}, {P, 0, 0}, {0, 0, 0}};
  const int smax = segs(512);
  for (int o = 0; o < 6; ++o) {
    for (int pab = M <= 255; pab >= 0; --pab) {
      for (int seg = smax; seg >= (smax > 4 ? 4 : smax); --seg) {
        const BLayout lo{seg, opts[o][0], opts[o][1], opts[o][2], pab};
        const size_t sm = bytes(lo, 4);
        if (sm <= cap) return run(lo, sm, false);
      }
    }
  }
  for (int seg = smax; seg >= 1; --seg) {   // the largest M accepted
    const BLayout lo{seg, 0, 0, 0, 0};
    const size_t sm = bytes(lo, 4);
    if (sm <= cap) return run(lo, sm, false);
  }
  return gpk::fail(GPK_EUNSUPPORTED, "psi_bwd: M=%d needs too much shared memory", M);
}

}  // namespace psi_impl
