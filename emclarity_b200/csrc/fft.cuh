// fft.cuh -- hand-written FP32 FFT building blocks for sm_100a.
//
// Register codelets of radix 2, 3, 4, 5, 7, 8, 12, 13 and 16, in two forms of a mixed-radix transform:
//
// * teams (fft_line, Stockham stages): a line in shared memory is transformed by P lanes of one warp (P
//   divides 32).  Each lane loads all the inputs of its butterflies into registers, the warp
//   synchronises, then the lane applies twiddles, runs the codelet and stores.  For contiguous lines: the
//   rows of the standalone transform and of the template search, the search's pass C.
// * lines across lanes (InPlace): neighbouring threads hold neighbouring lines and one butterfly each,
//   stages work in place, and only the exchanges between stages cross shared memory.  For strided axes:
//   k_cols, the template search's z pass; the search's passes A and B have their own two-stage variant.
//
// Sign convention: SIGN = -1 is the forward transform X_k = sum x_n e^{-2 pi i nk/L}
// (cuFFT / MATLAB fftn), SIGN = +1 the unnormalised inverse.
//
// Twiddles come from a per-length table tw[m] = exp(-2 pi i m / L), m in [0, L),
// computed on the host in double precision and rounded to float.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace emc {

__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__host__ __device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// a * (SIGN * i)
template <int SIGN>
__host__ __device__ __forceinline__ float2 mul_si(float2 a) {
  return SIGN < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

#ifdef __CUDACC__
// Pairs of FP32 values in one 64-bit register, and the packed multiply-add on them (sm_100): both
// components round to nearest like fmaf.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ unsigned long long fmul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long fadd2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// rounds towards minus infinity
__device__ __forceinline__ unsigned long long fadd2_rd(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

#endif
// a + b, a - b and a + s b (s real) of complex values by packed instructions on the device: the same
// roundings as the scalar forms in half the instructions (the arithmetic rate is the same, but the
// transforms' kernels are short of issue slots).
__host__ __device__ __forceinline__ float2 padd(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  return unpack2(fadd2(pack2(a.x, a.y), pack2(b.x, b.y)));
#else
  return cadd(a, b);
#endif
}
__host__ __device__ __forceinline__ float2 pfma(float2 a, float s, float2 b) {
#ifdef __CUDA_ARCH__
  return unpack2(ffma2(pack2(b.x, b.y), pack2(s, s), pack2(a.x, a.y)));
#else
  return make_float2(fmaf(b.x, s, a.x), fmaf(b.y, s, a.y));
#endif
}
__host__ __device__ __forceinline__ float2 psub(float2 a, float2 b) { return pfma(a, -1.f, b); }

// cos / sin of rational multiples of pi used inside the codelets (exact math constants).
#define EMC_SQRT1_2 0.70710678118654752440f
#define EMC_COS_PI8 0.92387953251128675613f
#define EMC_SIN_PI8 0.38268343236508977173f
#define EMC_SQRT3_2 0.86602540378443864676f

// ---------------------------------------------------------------- codelets
template <int R, int SIGN> struct Dft;

template <int SIGN> struct Dft<1, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2*) {}
};

template <int SIGN> struct Dft<2, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <int SIGN> struct Dft<3, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    float2 t1 = cadd(v[1], v[2]);
    float2 t2 = make_float2(fmaf(-0.5f, t1.x, v[0].x), fmaf(-0.5f, t1.y, v[0].y));
    float2 d = csub(v[1], v[2]);
    // i * SIGN * sqrt(3)/2 * d
    float2 t3 = mul_si<SIGN>(cscale(d, EMC_SQRT3_2));
    v[0] = cadd(v[0], t1);
    v[1] = cadd(t2, t3);
    v[2] = csub(t2, t3);
  }
};

template <int SIGN> struct Dft<4, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    float2 a0 = padd(v[0], v[2]), a1 = psub(v[0], v[2]);
    float2 b0 = padd(v[1], v[3]), b1 = mul_si<SIGN>(psub(v[1], v[3]));
    v[0] = padd(a0, b0);
    v[2] = psub(a0, b0);
    v[1] = cadd(a1, b1);  // (b1's components are swapped: no pair in registers)
    v[3] = csub(a1, b1);
  }
};

template <int SIGN> struct Dft<8, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    float2 e[4] = {v[0], v[2], v[4], v[6]};
    float2 o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, SIGN>::run(e);
    Dft<4, SIGN>::run(o);
    // w8^k = exp(SIGN 2 pi i k / 8); w8^1 o1 and w8^3 o3 without their factor 1 / sqrt 2
    float2 o1 = make_float2(o[1].x - (float)SIGN * o[1].y, o[1].y + (float)SIGN * o[1].x);
    float2 o2 = mul_si<SIGN>(o[2]);
    float2 o3 = make_float2(-o[3].x - (float)SIGN * o[3].y, -o[3].y + (float)SIGN * o[3].x);
    v[0] = padd(e[0], o[0]); v[4] = psub(e[0], o[0]);
    v[1] = pfma(e[1], EMC_SQRT1_2, o1); v[5] = pfma(e[1], -EMC_SQRT1_2, o1);
    v[2] = cadd(e[2], o2);   v[6] = csub(e[2], o2);
    v[3] = pfma(e[3], EMC_SQRT1_2, o3); v[7] = pfma(e[3], -EMC_SQRT1_2, o3);
  }
};

template <int SIGN> struct Dft<16, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    float2 e[8], o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { e[i] = v[2 * i]; o[i] = v[2 * i + 1]; }
    Dft<8, SIGN>::run(e);
    Dft<8, SIGN>::run(o);
    const float s = (float)SIGN;
    // w16^k = cos(2 pi k/16) + i SIGN sin(2 pi k/16)
    const float2 w[8] = {
        make_float2(1.f, 0.f),
        make_float2(EMC_COS_PI8, s * EMC_SIN_PI8),
        make_float2(EMC_SQRT1_2, s * EMC_SQRT1_2),
        make_float2(EMC_SIN_PI8, s * EMC_COS_PI8),
        make_float2(0.f, s),
        make_float2(-EMC_SIN_PI8, s * EMC_COS_PI8),
        make_float2(-EMC_SQRT1_2, s * EMC_SQRT1_2),
        make_float2(-EMC_COS_PI8, s * EMC_SIN_PI8)};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float2 t = (k == 0) ? o[0] : cmul(o[k], w[k]);
      v[k] = padd(e[k], t);
      v[k + 8] = psub(e[k], t);
    }
  }
};

// 12 = 3 x 4, coprime factors: with n = 4 n1 + 3 n2 and k = 4 k1 + 9 k2 (mod 12) the transform is three
// 4-point and four 3-point transforms without twiddles (Good, 1958).
template <int SIGN> struct Dft<12, SIGN> {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    float2 t[3][4];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < 4; ++n2) t[n1][n2] = v[(4 * n1 + 3 * n2) % 12];
      Dft<4, SIGN>::run(t[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      float2 u[3] = {t[0][k2], t[1][k2], t[2][k2]};
      Dft<3, SIGN>::run(u);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) v[(4 * k1 + 9 * k2) % 12] = u[k1];
    }
  }
};

// cos / sin(2 pi j / R) for the odd prime radices 5, 7 and 13 (exact values rounded to float).
__host__ __device__ constexpr float prime_cos(int R, int j) {
  return R == 5 ? (j == 0 ? 1.f : j == 1 ? 3.09016994374947451e-01f : j == 2 ? -8.09016994374947340e-01f
                 : j == 3 ? -8.09016994374947562e-01f : 3.09016994374947229e-01f)
       : R == 7 ? (j == 0 ? 1.f : j == 1 ? 6.23489801858733594e-01f : j == 2 ? -2.22520933956314337e-01f
                 : j == 3 ? -9.00968867902419035e-01f : j == 4 ? -9.00968867902419146e-01f
                 : j == 5 ? -2.22520933956314587e-01f : 6.23489801858733372e-01f)
                : (j == 0 ? 1.f : j == 1 ? 8.85456025653209911e-01f : j == 2 ? 5.68064746731155923e-01f
                 : j == 3 ? 1.20536680255323006e-01f : j == 4 ? -3.54604887042535455e-01f
                 : j == 5 ? -7.48510748171101192e-01f : j == 6 ? -9.70941817426052012e-01f
                 : j == 7 ? -9.70941817426052123e-01f : j == 8 ? -7.48510748171101303e-01f
                 : j == 9 ? -3.54604887042535899e-01f : j == 10 ? 1.20536680255323200e-01f
                 : j == 11 ? 5.68064746731154813e-01f : 8.85456025653210022e-01f);
}
__host__ __device__ constexpr float prime_sin(int R, int j) {
  return R == 5 ? (j == 0 ? 0.f : j == 1 ? 9.51056516295153531e-01f : j == 2 ? 5.87785252292473248e-01f
                 : j == 3 ? -5.87785252292473026e-01f : -9.51056516295153642e-01f)
       : R == 7 ? (j == 0 ? 0.f : j == 1 ? 7.81831482468029804e-01f : j == 2 ? 9.74927912181823619e-01f
                 : j == 3 ? 4.33883739117558231e-01f : j == 4 ? -4.33883739117558009e-01f
                 : j == 5 ? -9.74927912181823619e-01f : -7.81831482468029915e-01f)
                : (j == 0 ? 0.f : j == 1 ? 4.64723172043768507e-01f : j == 2 ? 8.22983865893656352e-01f
                 : j == 3 ? 9.92708874098053973e-01f : j == 4 ? 9.35016242685414833e-01f
                 : j == 5 ? 6.63122658240795193e-01f : j == 6 ? 2.39315664287557683e-01f
                 : j == 7 ? -2.39315664287557434e-01f : j == 8 ? -6.63122658240794971e-01f
                 : j == 9 ? -9.35016242685414722e-01f : j == 10 ? -9.92708874098053973e-01f
                 : j == 11 ? -8.22983865893657018e-01f : -4.64723172043768396e-01f);
}

// Odd prime radix: pairs (r, R-r) share the cosine term, X_q = x0 + sum_r [(x_r + x_{R-r}) cos
// + i SIGN (x_r - x_{R-r}) sin] with the angle 2 pi (q r mod R) / R.
template <int R, int SIGN>
struct DftPrime {
  static __host__ __device__ __forceinline__ void run(float2* v) {
    constexpr int H = (R - 1) / 2;
    float2 t1[H], t2[H];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      t1[r - 1] = cadd(v[r], v[R - r]);
      t2[r - 1] = csub(v[r], v[R - r]);
    }
    const float2 x0 = v[0];
    float2 s0 = x0;
#pragma unroll
    for (int r = 0; r < H; ++r) s0 = cadd(s0, t1[r]);
#pragma unroll
    for (int q = 1; q < R; ++q) {
      float2 acc = x0;
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const float c = prime_cos(R, (q * r) % R), s = (float)SIGN * prime_sin(R, (q * r) % R);
        acc.x = fmaf(t1[r - 1].x, c, fmaf(-t2[r - 1].y, s, acc.x));
        acc.y = fmaf(t1[r - 1].y, c, fmaf(t2[r - 1].x, s, acc.y));
      }
      v[q] = acc;
    }
    v[0] = s0;
  }
};
template <int SIGN> struct Dft<5, SIGN> : DftPrime<5, SIGN> {};
template <int SIGN> struct Dft<7, SIGN> : DftPrime<7, SIGN> {};
template <int SIGN> struct Dft<13, SIGN> : DftPrime<13, SIGN> {};

// ---------------------------------------------------------------- plans
// Generic plan for lengths without an explicit entry: radix-8 stages for the power of two (a 4
// or a 2 closes it), then 3s, 5s, 7s and 13s.  1 past the last stage, 0 for another prime factor.
__host__ __device__ constexpr int next_radix(int rem) {
  return rem % 8 == 0 ? 8 : rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : rem % 5 == 0 ? 5
       : rem % 7 == 0 ? 7 : rem % 13 == 0 ? 13 : 0;
}
__host__ __device__ constexpr int radix_seq_rem(int rem, int s) {
  return rem == 1 ? 1 : next_radix(rem) == 0 ? 0 : s == 0 ? next_radix(rem) : radix_seq_rem(rem / next_radix(rem), s - 1);
}
__host__ __device__ constexpr int radix_seq(int L, int s) { return L < 2 ? 0 : radix_seq_rem(L, s); }

// Radix sequence per supported length.  Stage s uses radix radix_of(L, s); 1 ends the plan.
__host__ __device__ constexpr int radix_of(int L, int s) {
  return L == 2   ? (s == 0 ? 2 : 1)
       : L == 3   ? (s == 0 ? 3 : 1)
       : L == 4   ? (s == 0 ? 4 : 1)
       : L == 6   ? (s == 0 ? 3 : s == 1 ? 2 : 1)
       : L == 8   ? (s == 0 ? 8 : 1)
       : L == 12  ? (s == 0 ? 4 : s == 1 ? 3 : 1)
       : L == 16  ? (s == 0 ? 16 : 1)
       : L == 24  ? (s == 0 ? 8 : s == 1 ? 3 : 1)
       : L == 32  ? (s == 0 ? 8 : s == 1 ? 4 : 1)
       : L == 48  ? (s == 0 ? 16 : s == 1 ? 3 : 1)
       : L == 64  ? (s == 0 ? 8 : s == 1 ? 8 : 1)
       : L == 96  ? (s == 0 ? 8 : s == 1 ? 4 : s == 2 ? 3 : 1)
       : L == 128 ? (s == 0 ? 16 : s == 1 ? 8 : 1)
       : L == 192 ? (s == 0 ? 8 : s == 1 ? 8 : s == 2 ? 3 : 1)
       : L == 256 ? (s == 0 ? 16 : s == 1 ? 16 : 1)
       : L == 384 ? (s == 0 ? 16 : s == 1 ? 8 : s == 2 ? 3 : 1)
       : L == 512 ? (s == 0 ? 8 : s == 1 ? 8 : s == 2 ? 8 : 1)
       // the remaining "nextBest" FFT sizes of coordinates/BH_multi_iterator.m:3-5 (factors 5, 7, 13)
       : radix_seq(L, s);
}

// Largest radix of a plan; used to pick a team size.
__host__ __device__ constexpr int max_radix(int L, int s = 0) {
  return radix_of(L, s) <= 1 ? 1
         : (radix_of(L, s) > max_radix(L, s + 1) ? radix_of(L, s) : max_radix(L, s + 1));
}
__host__ __device__ constexpr int min_butterflies(int L) { return radix_of(L, 0) == 0 ? 0 : L / max_radix(L); }

// Default team size: a power of two no larger than the smallest butterfly count, <= 32.
__host__ __device__ constexpr int team_size(int L) {
  return min_butterflies(L) >= 32 ? 32
       : min_butterflies(L) >= 16 ? 16
       : min_butterflies(L) >= 8  ? 8
       : min_butterflies(L) >= 4  ? 4
       : min_butterflies(L) >= 2  ? 2 : 1;
}

template <int SIGN>
__device__ __forceinline__ float2 twiddle(const float2* tw, int m) {
  float2 t = tw[m];
  return SIGN < 0 ? t : make_float2(t.x, -t.y);
}

// One Stockham stage of radix R on a line of length L; NS = product of earlier radices.
// buf: line base, elements at buf[i * stride].  Every lane of the warp must call this
// (inactive lanes pass active = false) because of the __syncwarp() calls.
// Physical slot of line element i.  With PAD, one spare slot follows every 8 elements: the
// radix-8 first stage writes elements 8j + r, which without the gap would put the 8 lanes of a
// team on 2 shared-memory banks.  padded_len(L) slots hold a padded line.
// PAD = 2 leaves the gap after every 16 elements instead, for lines whose first radix is 16
// (elements 16 j + r).
template <int PAD>
__host__ __device__ __forceinline__ constexpr int lpos(int i) {
  return PAD == 0 ? i : (PAD == 1 ? i + (i >> 3) : i + (i >> 4));
}
__host__ __device__ constexpr int padded_len(int L, int pad = 1) {
  return pad == 0 ? L : (pad == 1 ? L + L / 8 : L + L / 16);
}
// The padding that spreads the first stage's writes of a length-L line over the banks.  512
// (8 x 8 x 8) and 192 (8 x 8 x 3) also take the 16-element gap: their later stages read with
// strides of 64, where the 8-element gap leaves half-warps two or three ways on one bank (a
// half-warp model of the stage accesses gives 1.17 / 1.18 times the conflict-free wavefront
// count against 1.67 / 1.45 with the 8-element gap).
__host__ __device__ constexpr int line_pad(int L) {
  return radix_of(L, 0) >= 16 || L == 512 || L == 192 ? 2 : 1;
}

// Per-lane twiddles of stage S (NS = product of the earlier radices), kept in registers.  Lane
// `lane` of a team always handles butterflies j = lane + b P, whose twiddle exponents depend on
// k = j mod NS only -- not on which line the team transforms -- so a team can load them once
// and reuse them for every line.  Stages whose cache would exceed kTwCacheMax complex values
// (or that need no twiddles) read the shared-memory table instead.  The cache holds forward
// twiddles; inverse stages use their conjugates.
constexpr int kTwCacheMax = 8;

template <int L, int P, int S, int NS>
struct StageTw {
  static constexpr int R = radix_of(L, S);
  static constexpr int NB = L / R;
  static constexpr int PER = (NB + P - 1) / P;
  static constexpr bool kOn = NS > 1 && PER * (R - 1) <= kTwCacheMax;
  float2 w[kOn ? PER : 1][kOn ? R - 1 : 1];
  __device__ __forceinline__ void init(const float2* tw, int lane) {
    if constexpr (kOn) {
#pragma unroll
      for (int b = 0; b < PER; ++b) {
        const int k = (lane + b * P) % NS;
#pragma unroll
        for (int r = 1; r < R; ++r) w[b][r - 1] = tw[(r * k * (L / (NS * R))) % L];
      }
    }
  }
};

template <int L, int P, int S, int NS>
struct TwChain {
  StageTw<L, P, S, NS> st;
  TwChain<L, P, S + 1, NS * radix_of(L, S)> next;
  __device__ __forceinline__ void init(const float2* tw, int lane) {
    st.init(tw, lane);
    next.init(tw, lane);
  }
};
template <int L, int P, int S>
struct TwChain<L, P, S, L> {
  __device__ __forceinline__ void init(const float2*, int) {}
};

// Register twiddles of every stage of a length-L line transformed by teams of P lanes.
template <int L, int P = team_size(L)>
using LineTw = TwChain<L, P, 0, 1>;

// One Stockham stage of radix R on a line of length L (cache: optional register twiddles).
template <int L, int R, int NS, int SIGN, int P, int PAD, int S>
__device__ __forceinline__ void stockham_stage(float2* buf, int stride, int lane, const float2* tw,
                                               bool active, const StageTw<L, P, S, NS>* cache) {
  constexpr int NB = L / R;
  constexpr int PER = (NB + P - 1) / P;
  float2 v[PER][R];
#pragma unroll
  for (int b = 0; b < PER; ++b) {
    const int j = lane + b * P;
    if (active && (PER * P == NB || j < NB)) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[b][r] = buf[lpos<PAD>(j + r * NB) * stride];
    }
  }
  __syncwarp();
#pragma unroll
  for (int b = 0; b < PER; ++b) {
    const int j = lane + b * P;
    if (active && (PER * P == NB || j < NB)) {
      const int k = j % NS;
      if constexpr (NS > 1) {
        if constexpr (StageTw<L, P, S, NS>::kOn) {
          if (cache) {
#pragma unroll
            for (int r = 1; r < R; ++r)
              v[b][r] = SIGN < 0 ? cmul(v[b][r], cache->w[b][r - 1]) : cmulc(v[b][r], cache->w[b][r - 1]);
          } else {
#pragma unroll
            for (int r = 1; r < R; ++r) v[b][r] = cmul(v[b][r], twiddle<SIGN>(tw, (r * k * (L / (NS * R))) % L));
          }
        } else {
#pragma unroll
          for (int r = 1; r < R; ++r) v[b][r] = cmul(v[b][r], twiddle<SIGN>(tw, (r * k * (L / (NS * R))) % L));
        }
      }
      Dft<R, SIGN>::run(v[b]);
      const int idx = (j / NS) * NS * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) buf[lpos<PAD>(idx + r * NS) * stride] = v[b][r];
    }
  }
  __syncwarp();
}

template <int L, int SIGN, int P, int PAD, int S, int NS>
struct StageChain {
  static __device__ __forceinline__ void run(float2* buf, int stride, int lane, const float2* tw, bool active,
                                             const TwChain<L, P, S, NS>* tc) {
    constexpr int R = radix_of(L, S);
    stockham_stage<L, R, NS, SIGN, P, PAD, S>(buf, stride, lane, tw, active, tc ? &tc->st : nullptr);
    StageChain<L, SIGN, P, PAD, S + 1, NS * R>::run(buf, stride, lane, tw, active, tc ? &tc->next : nullptr);
  }
};
// terminate when the sub-transform length reaches L
template <int L, int SIGN, int P, int PAD, int S>
struct StageChain<L, SIGN, P, PAD, S, L> {
  static __device__ __forceinline__ void run(float2*, int, int, const float2*, bool, const TwChain<L, P, S, L>*) {}
};
// First stage (NS = 1, no twiddles) with its inputs produced by ld(i) -- element i of the line
// -- instead of loaded from the buffer, so a caller that builds the line (packing two real rows,
// Hermitian extension) skips one shared-memory round trip.
template <int L, int R, int SIGN, int P, int PAD, class Ld>
__device__ __forceinline__ void stockham_first_stage_in(const Ld& ld, float2* buf, int stride, int lane, bool active) {
  constexpr int NB = L / R;
  constexpr int PER = (NB + P - 1) / P;
  float2 v[PER][R];
#pragma unroll
  for (int b = 0; b < PER; ++b) {
    const int j = lane + b * P;
    if (active && (PER * P == NB || j < NB)) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[b][r] = ld(j + r * NB);
      Dft<R, SIGN>::run(v[b]);
#pragma unroll
      for (int r = 0; r < R; ++r) buf[lpos<PAD>(j * R + r) * stride] = v[b][r];
    }
  }
  __syncwarp();
}

// In-place complex FFT of one line held by a team of P lanes.  Element i lives at
// buf[lpos<PAD>(i) * stride].  tc (optional) holds the team lane's register twiddles.
template <int L, int SIGN, int P = team_size(L), int PAD = 0>
__device__ __forceinline__ void fft_line(float2* buf, int stride, int lane, const float2* tw, bool active,
                                         const LineTw<L, P>* tc = nullptr) {
  static_assert(radix_of(L, 0) != 0, "unsupported FFT length");
  static_assert(P >= 1 && P <= 32 && (32 % P) == 0, "team must divide a warp");
  StageChain<L, SIGN, P, PAD, 0, 1>::run(buf, stride, lane, tw, active, tc);
}

// FFT of a line whose elements come from ld(i) (see stockham_first_stage_in); the result is left
// in buf like fft_line's.
template <int L, int SIGN, int P = team_size(L), int PAD = 0, class Ld>
__device__ __forceinline__ void fft_line_in(const Ld& ld, float2* buf, int stride, int lane, const float2* tw,
                                            bool active, const LineTw<L, P>* tc = nullptr) {
  static_assert(radix_of(L, 0) != 0, "unsupported FFT length");
  constexpr int R0 = radix_of(L, 0);
  stockham_first_stage_in<L, R0, SIGN, P, PAD>(ld, buf, stride, lane, active);
  StageChain<L, SIGN, P, PAD, 1, R0>::run(buf, stride, lane, tw, active, tc ? &tc->next : nullptr);
}

// Number of stages of a length-L plan and the product of the radices before stage s.
__host__ __device__ constexpr int n_stages(int L, int s = 0) { return radix_of(L, s) <= 1 ? s : n_stages(L, s + 1); }
__host__ __device__ constexpr int radix_product(int L, int s) { return s == 0 ? 1 : radix_of(L, s - 1) * radix_product(L, s - 1); }

// ---------------------------------------------------------------- lines across lanes
// Mixed-radix stages for kernels whose neighbouring threads hold neighbouring lines: a thread has one
// butterfly of its own line at a time, so accesses are consecutive in the lines whatever the strides, and
// the stages work in place.  With M_s = L / (R_0 .. R_s), element n = sum r_s M_s starts at position n;
// stage s replaces digit r_s (stride M_s) by the output digit k_s, so that X(k_0 + R_0 k_1 + ..) ends at
// position sum k_s M_s, and the inverse over the same radices in reverse order ends in natural order.
// The butterflies, twiddles and their order are those of the Stockham stages above: same bits.
__host__ __device__ constexpr int digit_stride(int L, int s) { return L / radix_product(L, s + 1); }
// Output index k_0 + R_0 k_1 + .. held by the leading digits `hi` (k_0 most significant) of a position.
template <int L, int S>
__device__ __forceinline__ int digit_index(int hi) {
  if constexpr (S == 0) {
    return 0;
  } else if constexpr (S == 1) {
    return hi;
  } else {
    constexpr int R = radix_of(L, S - 1);
    return digit_index<L, S - 1>(hi / R) + radix_product(L, S - 1) * (hi % R);
  }
}
// Butterfly b of forward or (same radices, same order) inverse stage S: its first position and its
// index among the outputs formed so far.
template <int L, int S>
struct InPlace {
  static constexpr int R = radix_of(L, S), M = digit_stride(L, S), NS = radix_product(L, S), NB = L / R;
  static __device__ __forceinline__ int base(int b) { return (b / M) * (R * M) + b % M; }
  static __device__ __forceinline__ int index(int b) { return digit_index<L, S>(b / M); }
  // twiddles of a loaded butterfly, then its transform
  template <int SIGN>
  static __device__ __forceinline__ void run(float2 (&v)[R], int k, const float2* tw) {
    if constexpr (NS > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], twiddle<SIGN>(tw, r * k * (L / (NS * R))));
    }
    Dft<R, SIGN>::run(v);
  }
};

// Loads the length-L twiddle table into shared memory (cooperatively, whole block).
template <int L>
__device__ __forceinline__ void load_twiddles(float2* s_tw, const float2* g_tw) {
  for (int i = threadIdx.x + threadIdx.y * blockDim.x; i < L; i += blockDim.x * blockDim.y) s_tw[i] = g_tw[i];
}

// Map a float to an unsigned key with the same order (for atomicMax-based argmax).
__device__ __forceinline__ uint32_t ordered_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float key_to_float(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}

}  // namespace emc
