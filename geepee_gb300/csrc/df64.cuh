// Double-float ("df64") arithmetic on the FP32 pipes of sm_103a.
//
// A value is the unevaluated sum hi + lo of two floats (|lo| <= ulp(hi)/2), giving
// about 48 significant bits.  GB300 issues FP32 FMAs at ~60x its FP64 rate, so the
// error-free transformations below (Knuth two-sum, FMA two-product) buy FP64-class
// accuracy for the ill-conditioned parts of the sparse-GP path at a fraction of the
// cost of native double.  Algorithms: Dekker/Knuth error-free transforms and the
// double-double scheme of Hida, Li & Bailey ("Algorithms for quad-double precision
// floating point arithmetic", ARITH 2001), specialised to float pairs.
//
// The same kernels are instantiated for plain `float`; the overload set below lets
// templated code be written once (add/mul/fma_/exp_/...).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct __align__(8) df64 {   // 8-byte alignment: an element in memory is one access
  float hi, lo;
};

__host__ __device__ __forceinline__ df64 make_df(float h, float l = 0.f) { df64 r; r.hi = h; r.lo = l; return r; }

// float64 -> (hi, lo): hi = x rounded to float, lo = (x - hi) rounded to float, by integer operations
// on the bit pattern: the FP64 pipe, which the plain conversion would use, issues ~64x slower than
// the integer pipes on this part.  hi is the pattern rounded to 24 bits (nearest even) with its
// exponent field lowered; lo is the remainder, at most 2^28 units of x's last place, converted by the
// 32-bit conversion (the same rounding) with its exponent field lowered: ~16 instructions where
// normalising and rounding the remainder by hand took 45.  Zeros, and values whose lo could
// be subnormal or hi not a normal float (|x| < 2^-74 or >= 2^128, inf, nan), are left to
// df_from_double_rest, out of line: inlined, the compiler if-converts the rare branch and runs its
// instructions for every conversion.
static __device__ __noinline__ df64 df_from_double_fp64(double x) {
  float h = __double2float_rn(x);
  float l = __double2float_rn(x - (double)h);
  return make_df(h, l);
}
// the same with every rounding step in integers, for any normal hi (lo may come out subnormal); the
// FP64 path for the rest
static __device__ __noinline__ df64 df_from_double_rest(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  if ((b << 1) == 0ull) return make_df(__int_as_float((int)(b >> 32)), 0.f);   // +-0
  if (e < 897 || e > 1150) return df_from_double_fp64(x);   // hi would be subnormal / inf / nan
  const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  unsigned top = (unsigned)(mant >> 29);
  int rem = (int)(mant & 0x1FFFFFFFull);
  if (rem > 0x10000000 || (rem == 0x10000000 && (top & 1u))) {
    top += 1u;
    rem -= 0x20000000;
  }
  int fe = e - 1023 + 127;
  if (top == 0x1000000u) {
    top >>= 1;
    fe += 1;
  }
  const unsigned sign = (unsigned)(b >> 63);
  const float hi = __uint_as_float((sign << 31) | ((unsigned)fe << 23) | (top & 0x7fffffu));
  float lo = 0.f;
  if (rem != 0) {
    unsigned rs = 0u;
    unsigned r = (unsigned)rem;
    if (rem < 0) {
      rs = 1u;
      r = (unsigned)(-rem);
    }
    const int nb = 32 - __clz(r);
    int sh = nb - 24;
    const unsigned ls = (sign ^ rs) << 31;
    const int le0 = e - 1075 + sh + 23 + 127;   // lo's exponent field before rounding
    if (le0 >= 1) {
      unsigned m;
      if (sh > 0) {
        m = r >> sh;
        const unsigned rem2 = r & ((1u << sh) - 1u), half = 1u << (sh - 1);
        if (rem2 > half || (rem2 == half && (m & 1u))) ++m;
        if (m == 0x1000000u) {
          m >>= 1;
          ++sh;
        }
      } else {
        m = r << (-sh);
      }
      const int le = e - 1075 + sh + 23 + 127;
      lo = __uint_as_float(ls | ((unsigned)le << 23) | (m & 0x7fffffu));
    } else {
      // subnormal lo: round the remainder once, straight to the subnormal's precision (a
      // carry into bit 23 gives the smallest normal, which the bit pattern encodes as is)
      const int t = sh + 1 - le0;
      unsigned q = 0u;
      if (t <= 0) {
        q = r << (-t);
      } else if (t < 32) {
        q = r >> t;
        const unsigned rr = r & ((1u << t) - 1u), hf = 1u << (t - 1);
        if (rr > hf || (rr == hf && (q & 1u))) ++q;
      }
      lo = __uint_as_float(ls | q);
    }
  }
  return make_df(hi, lo);
}
// whether df_from_double_plain does for x: zero, or in the range above
__device__ __forceinline__ bool df_plain(double x) {
  const unsigned hw = (unsigned)__double2hiint(x);
  return ((hw >> 20) & 0x7ff) - 949u <= 201u || ((hw << 1) | (unsigned)__double2loint(x)) == 0u;
}
__device__ __forceinline__ df64 df_from_double_plain(double x) {
  const unsigned hw = (unsigned)__double2hiint(x), lw = (unsigned)__double2loint(x);
  const int e = (int)((hw >> 20) & 0x7ff);
  const unsigned long long m = ((unsigned long long)(hw & 0x7fffffffu) << 32) | lw;
  const unsigned top = (unsigned)((m + 0x0fffffffull + ((m >> 29) & 1u)) >> 29);   // (mod 2^32: the field's excess)
  const float g = (float)(int)(lw - (top << 29));
  const unsigned lo = g == 0.f ? 0u : (__float_as_uint(g) + ((unsigned)(e - 1075) << 23)) ^ (hw & 0x80000000u);
  return make_df(e == 0 ? 0.f : __uint_as_float((top - (896u << 23)) | (hw & 0x80000000u)), __uint_as_float(lo));
}
__device__ __forceinline__ df64 df_from_double(double x) {
  const unsigned hw = (unsigned)__double2hiint(x), lw = (unsigned)__double2loint(x);
  const int e = (int)((hw >> 20) & 0x7ff);
  if (e < 949 || e > 1150) {
    if (((hw << 1) | lw) == 0u) return make_df(__int_as_float((int)hw), 0.f);   // +-0
    return df_from_double_rest(x);
  }
  return df_from_double_plain(x);
}
__device__ __forceinline__ double df_to_double(df64 a) { return (double)a.hi + (double)a.lo; }

// ---- error-free transforms ----
__device__ __forceinline__ df64 two_sum(float a, float b) {
  float s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return make_df(s, e);
}
__device__ __forceinline__ df64 quick_two_sum(float a, float b) {  // |a| >= |b|
  float s = __fadd_rn(a, b);
  float e = __fsub_rn(b, __fsub_rn(s, a));
  return make_df(s, e);
}
__device__ __forceinline__ df64 two_prod(float a, float b) {
  float p = __fmul_rn(a, b);
  float e = __fmaf_rn(a, b, -p);
  return make_df(p, e);
}

// ---- arithmetic ----
// "sloppy" double-float add (Hida-Li-Bailey): error <= ~2^-47 (|a| + |b|), the same
// shape of bound as an FP64 add; 11 FP32 ops.
__device__ __forceinline__ df64 add(df64 a, df64 b) {
  df64 s = two_sum(a.hi, b.hi);
  s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  return quick_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df64 neg(df64 a) { return make_df(-a.hi, -a.lo); }
__device__ __forceinline__ df64 sub(df64 a, df64 b) { return add(a, neg(b)); }
__device__ __forceinline__ df64 add(df64 a, float b) {
  df64 s = two_sum(a.hi, b);
  s.lo = __fadd_rn(s.lo, a.lo);
  return quick_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df64 mul(df64 a, df64 b) {
  df64 p = two_prod(a.hi, b.hi);
  p.lo = __fmaf_rn(a.hi, b.lo, p.lo);
  p.lo = __fmaf_rn(a.lo, b.hi, p.lo);
  return quick_two_sum(p.hi, p.lo);
}
__device__ __forceinline__ df64 mul(df64 a, float b) {
  df64 p = two_prod(a.hi, b);
  p.lo = __fmaf_rn(a.lo, b, p.lo);
  return quick_two_sum(p.hi, p.lo);
}
// a*b + c: the product's exact high part (FMA two-product) and its cross terms go into one
// sloppy double-float addition with c, without normalising the product first (14 FP32 ops
// instead of 17; error bound of the same shape, ~2^-47 (|a b| + |c|)).
__device__ __forceinline__ df64 fma_(df64 a, df64 b, df64 c) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  df64 s = two_sum(c.hi, p);
  s.lo = __fadd_rn(s.lo, __fadd_rn(c.lo, e));
  return quick_two_sum(s.hi, s.lo);
}
// 2^e as a float for e in [-126, 127] (built from the exponent field: no conversion unit)
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
// a * 2^e, exact while the results stay normal: one multiply for |e| <= 126 (constant e folds
// to it), two for |e| <= 252 (the range exp_tab needs)
__device__ __forceinline__ float scale2f(float a, int e) {
  if (e >= -126 && e <= 127) return a * pow2f(e);
  const int e1 = e >> 1;
  return a * pow2f(e1) * pow2f(e - e1);
}
__device__ __forceinline__ df64 scale2(df64 a, int e) { return make_df(scale2f(a.hi, e), scale2f(a.lo, e)); }

__device__ __forceinline__ df64 div(df64 a, df64 b) {
  float q1 = __fdiv_rn(a.hi, b.hi);
  df64 r = sub(a, mul(b, q1));
  float q2 = __fdiv_rn(r.hi, b.hi);
  r = sub(r, mul(b, q2));
  float q3 = __fdiv_rn(r.hi, b.hi);
  df64 q = quick_two_sum(q1, q2);
  return add(q, q3);
}
__device__ __forceinline__ df64 recip(df64 b) { return div(make_df(1.f), b); }

// sqrt by one Newton correction of the float root: s + (a - s^2) / (2 s)
__device__ __forceinline__ df64 sqrt_(df64 a) {
  if (a.hi <= 0.f) return make_df(0.f);
  float s = sqrtf(a.hi);
  df64 r = sub(a, two_prod(s, s));
  float c = __fdiv_rn(r.hi, 2.f * s);
  return quick_two_sum(s, c);
}

// 1/sqrt(a), a > 0: the float estimate y corrected by the binomial series of (1 - h)^(-1/2),
//   1/sqrt(a) = y (1 + h/2 + 3 h^2/8 + ...),  h = 1 - a y^2,
// where a y^2 is formed in double-float, h = hh + hl is kept as an unevaluated pair (1 - t.hi
// is exact, |h| ~ 2^-22) and the leading correction y hh is an exact product, so that only
// terms below 2^-46 y are rounded in single precision.  The omitted 5 h^3/16 is ~2^-64.
// Measured on a CPU emulation of these operations (20000 inputs over e^[-10,10], estimates
// perturbed by up to 2 ulp): relative error <= 2^-47.1, mean 2^-50.
__device__ __forceinline__ df64 rsqrt_(df64 a) {
  const float y = rsqrtf(a.hi);
  const df64 t = mul(a, two_prod(y, y));
  const float hh = __fsub_rn(1.f, t.hi), hl = -t.lo;
  const float h = __fadd_rn(hh, hl);
  const df64 c = two_prod(y, hh);
  float rest = __fmaf_rn(y, hl, c.lo);
  rest = __fmaf_rn(__fmul_rn(__fmul_rn(y, h), h), 0.75f, rest);   // y (hl + 3/4 h^2) + the product's tail
  df64 r = quick_two_sum(y, __fmul_rn(c.hi, 0.5f));
  r.lo = __fmaf_rn(rest, 0.5f, r.lo);
  return quick_two_sum(r.hi, r.lo);
}

// ---- exp: table-driven reduction x = k ln2/256 + r, |r| <= ln2/512 ----
// Table T[j] = 2^(j/256) stored as df64 (exp2_table.cuh); copied into shared memory
// once per CTA by load_exp_table().
#define GPK_EXP_TABLE 256
#include "exp2_table.cuh"

// ln2/256 = 0.0027076061740622863 as a df64 (hi + lo exact to 3.4e-19)
__device__ __forceinline__ df64 ln2_over_256() { return make_df(2.707606182e-03f, -7.440055516e-12f); }

// NARROW: the domain [-87, 88]; below it the result (< 1.6e-38, already subnormal in its high
// word) is flushed to zero, so that the final scaling 2^m has m in [-126, 126] and takes one
// multiply per word instead of the two-step range-checked one
template <bool NARROW = false, typename Tab>
__device__ __forceinline__ df64 exp_tab(df64 x, const Tab& tab) {
  if (x.hi < (NARROW ? -87.0f : -103.0f)) return make_df(0.f);
  if (x.hi > 88.0f) return make_df(__int_as_float(0x7f800000), 0.f);
  const float inv = 369.32993f;  // 256 / ln 2
  // k = round(x / (ln2/256)) by the 1.5*2^23 magic addition (|x * inv| < 2^22 here): the
  // rounding and the integer both come from one FP32 add, with no conversion instruction
  const float kb = __fadd_rn(x.hi * inv, 12582912.f);
  const float kf = __fsub_rn(kb, 12582912.f);
  const int k = __float_as_int(kb) - 0x4B400000;
  df64 r = sub(x, mul(ln2_over_256(), kf));
  // exp(r) - 1 = r + r^2/2 + r^3/6 + r^4/24  (|r| < 1.4e-3; next term < 4e-17)
  df64 r2 = mul(r, r);
  float t = r.hi * r2.hi * (0.16666667f + r.hi * 0.041666668f);
  df64 p = add(add(r, scale2(r2, -1)), t);
  df64 e = add(p, 1.0f);
  int j = k & (GPK_EXP_TABLE - 1);
  int m = k >> 8;  // arithmetic shift: floor(k / 256)
  float2 tj = tab[j];
  df64 res = mul(make_df(tj.x, tj.y), e);
  if (NARROW) {
    const float s2m = pow2f(m);
    return make_df(res.hi * s2m, res.lo * s2m);
  }
  return scale2(res, m);
}

// ---- exp2 of a fixed-point argument (the psi2 pair sweeps) ----
// x is a base-2 exponent in units of 2^-52, plus the half step 2^-12 that centres the table
// reduction (the caller folds kFxHalf into one of x's terms).  The table T[j] = 2^(j/2048) takes
// x's top 11 fraction bits, so that the remainder r, |r| <= 2^-12, needs only the first-order term
// in two floats: 2^r - 1 = p + p^2/2 + p^3/6, p = r ln 2 < 1.7e-4, whose p^2/2 < 2^-26 is exact to
// 2^-50 in one float.  ~30 instructions where the double-float argument reduction and polynomial
// of exp_tab take ~80, and the argument's sums are integer additions (2 instructions instead
// of 11).  Results below 2^-126 are flushed to zero; x must be below 127 * 2^52.
constexpr int kFxTab = 2048;
constexpr long long kFxHalf = 1LL << 40;
// T[j], j < 2048, from the 256-entry table: T[8 j + i] = 2^(j/256) 2^(i/2048); 2^(i/2048) - 1 as
// double-float constants (60-digit decimal arithmetic, rounded as in exp2_table.cuh)
__device__ __forceinline__ void load_exp2_table(float2* s_tab) {
  const float c_hi[8] = {0.000000000e+00f, 3.385080490e-04f, 6.771307089e-04f, 1.015867922e-03f, 1.354719861e-03f, 1.693686470e-03f, 2.032767981e-03f, 2.371964045e-03f};
  const float c_lo[8] = {0.000000000e+00f, 3.656181261e-12f, -1.587024435e-11f, 3.841724161e-11f, 3.069764928e-11f, 5.799375910e-11f, -7.369679866e-11f, 2.371333858e-11f};
  // a warp's 32 consecutive entries need four of the 256; eight rounds' worth arrive by one load a lane (a load in
  // each round made the table ~2 us of a launch)
  const int lane = threadIdx.x & 31, first = threadIdx.x & ~31, i = lane & 7;
  float ch = 0.f, cl = 0.f;
#pragma unroll
  for (int u = 1; u < 8; ++u) {
    ch = i == u ? c_hi[u] : ch;
    cl = i == u ? c_lo[u] : cl;
  }
#pragma unroll 1
  for (int b = first; b < kFxTab; b += 8 * blockDim.x) {
    const int j = ((b + (lane >> 2) * (int)blockDim.x) >> 3) + (lane & 3);
    const float2 all = j < 256 ? kExp2Tab[j] : make_float2(0.f, 0.f);
    float2* const out = s_tab + b + lane;
#pragma unroll 1
    for (int r = 0; r < 8 && b + r * (int)blockDim.x < kFxTab; ++r) {
      const float2 t = make_float2(__shfl_sync(0xffffffffu, all.x, 4 * r + (lane >> 3)),
                                   __shfl_sync(0xffffffffu, all.y, 4 * r + (lane >> 3)));
      // t (1 + c): the product's exact high part and its cross terms added to t
      const df64 w = two_prod(t.x, ch);
      const float e = __fadd_rn(__fmaf_rn(t.x, cl, w.lo), __fmaf_rn(t.y, ch, t.y));
      df64 q = quick_two_sum(t.x, w.hi);
      q = quick_two_sum(q.hi, __fadd_rn(q.lo, e));
      out[r * blockDim.x] = make_float2(q.hi, q.lo);
    }
  }
}
// the 256-entry exp table of exp_tab inside that table (every 8th entry)
struct ExpTab {
  const float2* p;
  __device__ __forceinline__ float2 operator[](int j) const { return p[8 * j]; }
};
// 2^(x's fraction) as h + l, h in (0.999, 2); tab: the table's shared-memory address
__device__ __forceinline__ df64 exp2_fx_frac(long long x, unsigned tab) {
  const unsigned xl = (unsigned)x;
  const int xh = (int)(x >> 32);
  float2 T;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(T.x), "=f"(T.y) : "r"(tab + ((xh >> 6) & ((kFxTab - 1) << 3))));
  // the 41 remainder bits as two floats, by exponent splicing: 23 bits of [1, 2), then 18
  const float f = __uint_as_float(0x3f800000u | (__funnelshift_l(xl, (unsigned)xh, 14) & 0x7fffffu));
  const float g = __uint_as_float(0x4b000000u | (xl & 0x3ffffu));   // 2^23 + the low 18 bits
  const float a = __fsub_rn(f, 1.5f);                               // r = a 2^-11 + (low bits) 2^-52
  const float c1 = 3.384507727e-04f, c1l = -9.300069395e-13f, c2 = 1.539095923e-16f;                // ln2 2^-11 (hi, lo), ln2 2^-52
  const float p = __fmul_rn(a, c1);
  float t = __fmaf_rn(g, c2, -8388608.f * c2);
  t = __fmaf_rn(a, c1l, t);
  float e = __fadd_rn(t, __fmaf_rn(a, c1, -p));
  e = __fmaf_rn(p, e, e);
  e = __fmaf_rn(__fmul_rn(p, p), __fmaf_rn(p, 0.16666667f, 0.5f), e);   // 2^r = 1 + p + e
  // T 2^r, then 2^m by one multiply a word
  const float w = __fmul_rn(T.x, p);
  float l = __fmaf_rn(T.x, e, __fmaf_rn(T.x, p, -w));
  l = __fadd_rn(l, __fmaf_rn(T.y, p, T.y));
  const float h = __fadd_rn(T.x, w);
  l = __fadd_rn(l, __fsub_rn(w, __fsub_rn(h, T.x)));
  return make_df(h, l);
}
__device__ __forceinline__ df64 exp2_fx(long long x, unsigned tab) {
  const df64 r = exp2_fx_frac(x, tab);
  const int xh = (int)(x >> 32);
  const float s = xh >= -(126 << 20) ? __int_as_float(((xh << 3) & 0xff800000) + 0x3f800000) : 0.f;
  return make_df(__fmul_rn(r.hi, s), __fmul_rn(r.lo, s));
}
// the same as a float64, by integer operations: h's bits widened, l added in units of h's last
// float64 place (below 1 the unit halves; h = 1 with a negative l counts as below)
// results below 2^MINE are flushed to zero
template <int MINE = -126>
__device__ __forceinline__ double exp2_fx_double(long long x, unsigned tab) {
  const df64 r = exp2_fx_frac(x, tab);
  const int xh = (int)(x >> 32);
  const bool below = r.hi < 1.f || (r.hi == 1.f && r.lo < 0.f);
  const int li = __float2int_rn(__fmul_rn(r.lo, below ? 9007199254740992.f : 4503599627370496.f));
  const unsigned hb = __float_as_uint(r.hi);
  long long d = ((long long)hb << 29) + ((896LL + (xh >> 20)) << 52) + li;
  return __longlong_as_double(xh >= MINE * (1 << 20) ? d : 0LL);
}
// x 2^F truncated to an integer (|x 2^F| < 2^63, the exponent field at most 189 - F), by shifting
// the significand: the float-to-64-bit-integer conversion issues on the FP64 pipe, 16 cycles a warp
template <int F>
__device__ __forceinline__ long long fx_bits(float x) {
  const unsigned b = __float_as_uint(x);
  const int s = min(189 - F - (int)((b >> 23) & 0xffu), 63);
  const long long v = (long long)(((unsigned long long)(((b & 0x7fffffu) | 0x800000u) << 7) << 32) >> s);
  return (int)b < 0 ? -v : v;
}
// a double-float in units of 2^-52 (|v| < 1024)
__device__ __forceinline__ long long fx52_of(df64 v) { return fx_bits<52>(v.hi) + fx_bits<52>(v.lo); }
// a double-float (|v| < 16) as two words, high 2^-26 + low 2^-57 with |low| <= 2^30
__device__ __forceinline__ long long fx57_words_of(df64 v) {
  const long long t = fx_bits<57>(v.hi) + fx_bits<57>(v.lo) + (1LL << 30);
  const int high = (int)(t >> 31), low = (int)((unsigned)t & 0x7fffffffu) - (1 << 30);
  return ((long long)high << 32) | (unsigned)low;
}
// hi + lo as a float64 by integer operations (df_to_double's three FP64-pipe instructions take 48
// cycles a warp): hi's bits widened, lo added in units of hi's last float64 place (half of it
// below a power of two).  Values whose words leave the normal range take the FP64 path.
__device__ __forceinline__ double df_to_double_int(df64 a) {
  const unsigned hb = __float_as_uint(a.hi), lb = __float_as_uint(a.lo);
  const int he = (int)((hb >> 23) & 0xffu), le = (int)((lb >> 23) & 0xffu);
  const bool against = (int)(hb ^ lb) < 0;                          // lo takes away from |hi|
  const int k = 127 + 52 + (((hb & 0x7fffffu) == 0u && against) ? 1 : 0) - he;   // lo 2^k: exponent field le + k
  if (he == 0 || he == 255 || (le == 0 && (lb << 1) != 0u) || le + k > 158) return df_to_double(a);
  const int li = le == 0 || le + k < 1 ? 0 : __float2int_rn(__uint_as_float((lb & 0x7fffffu) | ((unsigned)(le + k) << 23)));
  const long long mag = ((long long)(hb & 0x7fffffffu) << 29) + (896LL << 52) + (against ? -li : li);
  return __longlong_as_double(mag | ((long long)(hb & 0x80000000u) << 32));
}

// log2(e) in the precision of the argument
__device__ __forceinline__ df64 log2e_of(df64) { return make_df(1.442695022e+00f, 1.925963034e-08f); }

// the storage value of a compute value by integer operations (see df_to_double_int)
__device__ __forceinline__ double st_int(df64 a) { return df_to_double_int(a); }
__device__ __forceinline__ double st_int(float a) { return (double)a; }

// log by one Newton step on exp: y1 = y0 + x exp(-y0) - 1
template <typename Tab>
__device__ __forceinline__ df64 log_tab(df64 x, const Tab& tab) {
  float y0 = logf(x.hi);
  df64 ey = exp_tab(make_df(-y0), tab);
  df64 c = sub(mul(x, ey), make_df(1.f));
  return add(make_df(y0), c);
}

// ---- warp reductions ----
__device__ __forceinline__ df64 shfl_xor(df64 a, int m) {
  return make_df(__shfl_xor_sync(0xffffffffu, a.hi, m), __shfl_xor_sync(0xffffffffu, a.lo, m));
}
__device__ __forceinline__ float shfl_xor(float a, int m) { return __shfl_xor_sync(0xffffffffu, a, m); }
__device__ __forceinline__ df64 shfl_idx(df64 a, int src) {
  return make_df(__shfl_sync(0xffffffffu, a.hi, src), __shfl_sync(0xffffffffu, a.lo, src));
}
__device__ __forceinline__ float shfl_idx(float a, int src) { return __shfl_sync(0xffffffffu, a, src); }
__device__ __forceinline__ df64 warp_sum(df64 a) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) a = add(a, shfl_xor(a, m));
  return a;
}
__device__ __forceinline__ float warp_sum(float a) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) a += __shfl_xor_sync(0xffffffffu, a, m);
  return a;
}
// ---- float overloads so templated kernels compile for T = float ----
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ float sub(float a, float b) { return a - b; }
__device__ __forceinline__ float mul(float a, float b) { return a * b; }
__device__ __forceinline__ float neg(float a) { return -a; }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float recip(float b) { return __fdiv_rn(1.f, b); }
__device__ __forceinline__ float sqrt_(float a) { return sqrtf(fmaxf(a, 0.f)); }
__device__ __forceinline__ float rsqrt_(float a) { return __frsqrt_rn(a); }
__device__ __forceinline__ float scale2(float a, int e) { return scale2f(a, e); }
template <typename Tab> __device__ __forceinline__ float exp_tab(float x, const Tab&) { return expf(x); }
template <typename Tab> __device__ __forceinline__ float log_tab(float x, const Tab&) { return logf(x); }
// The exp of the psi2 pair sweeps' rare path (arguments outside the fixed-point range)
template <typename Tab> __device__ __forceinline__ df64 exp_pair(df64 x, const Tab& tab) { return exp_tab<true>(x, tab); }
template <typename Tab> __device__ __forceinline__ float exp_pair(float x, const Tab&) { return __expf(x); }

__device__ __forceinline__ float log2e_of(float) { return 1.44269504f; }
// a b + c of 32-bit factors in one instruction (from C, the compiler widens the factors to 64 bits
// first: three multiply-adds and two shifts a product)
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// max that returns NaN when either is NaN
__device__ __forceinline__ float fmax_nan(float a, float b) { return (a != a || b != b) ? __int_as_float(0x7fffffff) : fmaxf(a, b); }

// a running sum kept as (hi, lo) without renormalising: for sums of a few dozen terms (the low
// word's own rounding stays below the normalised sum's)
__device__ __forceinline__ void acc_add(df64& a, df64 x) {
  const df64 s = two_sum(a.hi, x.hi);
  a.hi = s.hi;
  a.lo = __fadd_rn(a.lo, __fadd_rn(s.lo, x.lo));
}
__device__ __forceinline__ void acc_fma(df64& a, df64 x, df64 y) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -p);
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  const df64 s = two_sum(a.hi, p);
  a.hi = s.hi;
  a.lo = __fadd_rn(a.lo, __fadd_rn(s.lo, e));
}
__device__ __forceinline__ df64 acc_done(df64 a) { return quick_two_sum(a.hi, a.lo); }
__device__ __forceinline__ void acc_add(float& a, float x) { a += x; }
__device__ __forceinline__ void acc_fma(float& a, float x, float y) { a = __fmaf_rn(x, y, a); }
__device__ __forceinline__ float acc_done(float a) { return a; }

// Warp sums of K values at once (K a power of two <= 32): in each of the first log2 K steps
// of the butterfly a lane keeps half of its values and adds its partner's copies of them,
// trading the other half, so the K sums take K - 1 + 5 - log2 K exchanges instead of 5 K.
// On return v[0] of lane l holds the warp total of value l >> (5 - log2 K).
template <int K, typename T>
__device__ __forceinline__ void warp_sum_many(T (&v)[K]) {
  static_assert(K >= 1 && K <= 32 && (K & (K - 1)) == 0, "K must be a power of two <= 32");
  const int lane = threadIdx.x & 31;
  int off = 16;
#pragma unroll
  for (int n = K; n > 1; n >>= 1, off >>= 1) {
    const bool up = (lane & off) != 0;   // this lane keeps the upper half of the n values
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const T keep = up ? v[i + n / 2] : v[i];
      const T send = up ? v[i] : v[i + n / 2];
      v[i] = add(keep, shfl_xor(send, off));
    }
  }
#pragma unroll
  for (; off > 0; off >>= 1) v[0] = add(v[0], shfl_xor(v[0], off));
}

// conversions between storage (double / float) and compute (df64 / float) types
template <typename T> struct Num;
template <> struct Num<df64> {
  typedef double store_t;
  __device__ static __forceinline__ df64 ld(double x) { return df_from_double(x); }
  __device__ static __forceinline__ double st(df64 x) { return df_to_double(x); }
  __device__ static __forceinline__ df64 c(float x) { return make_df(x); }
  __device__ static __forceinline__ df64 zero() { return make_df(0.f); }
  __device__ static __forceinline__ float approx(df64 x) { return x.hi; }
};
template <> struct Num<float> {
  typedef float store_t;
  __device__ static __forceinline__ float ld(float x) { return x; }
  __device__ static __forceinline__ float st(float x) { return x; }
  __device__ static __forceinline__ float c(float x) { return x; }
  __device__ static __forceinline__ float zero() { return 0.f; }
  __device__ static __forceinline__ float approx(float x) { return x; }
};

// the exp table lives in shared memory; every kernel that calls exp_tab loads it first
__device__ __forceinline__ void load_exp_table(float2* s_tab) {
  for (int i = threadIdx.x; i < GPK_EXP_TABLE; i += blockDim.x) s_tab[i] = kExp2Tab[i];
}
