// fft_passes.cuh -- generic single-axis FFT passes over global memory.
//
// These are the building blocks of the standalone R2C / C2R transform (the mexFFT
// replacement), of the particle-spectrum preparation and of the large-volume
// template search.  The fused orientation-search kernels use the same line FFT
// but keep the data on chip between axes.
#pragma once
#include "common.cuh"

namespace emc {

// ----------------------------------------------------------------- rows, R2C
// nrows real rows of length L (pitch in_pitch floats) -> complex rows of length
// L/2+1 (pitch out_pitch float2).  Two rows share one complex FFT: z = a + i b.
// Teams per CTA of the row kernels: at most 256 threads and ~32 KB of line buffers.
// Line buffers hold padded lines (lpos<line_pad(L)>, see fft.cuh) against bank conflicts.
__host__ __device__ constexpr int row_line_len(int L) { return padded_len(L, line_pad(L)) + 1; }
__host__ __device__ constexpr int rows_teams(int L, int P) {
  return (256 / P) < (4096 / row_line_len(L)) ? (256 / P)
                                               : ((4096 / row_line_len(L)) > 0 ? (4096 / row_line_len(L)) : 1);
}

template <int L, int P>
__global__ void __launch_bounds__(256) k_rows_r2c(const float* __restrict__ in, long in_pitch,
                                                  float2* __restrict__ out, long out_pitch, long nrows,
                                                  const float2* __restrict__ g_tw) {
  constexpr int TEAMS = rows_teams(L, P);
  constexpr int PAD = line_pad(L);
  __shared__ float2 s_tw[L];
  __shared__ float2 s_line[TEAMS][row_line_len(L)];
  load_twiddles<L>(s_tw, g_tw);
  __syncthreads();
  const int team = threadIdx.x / P, lane = threadIdx.x % P;
  const long npairs = (nrows + 1) / 2;
  for (long pair0 = (long)blockIdx.x * TEAMS; pair0 < npairs; pair0 += (long)gridDim.x * TEAMS) {
    const long pair = pair0 + team;
    const bool active = pair < npairs;
    const long ra = 2 * pair, rb = 2 * pair + 1;
    const bool has_b = rb < nrows;
    float2* buf = s_line[team];
    const float* a = in + ra * in_pitch;
    const float* b = in + rb * in_pitch;
    fft_line_in<L, -1, P, PAD>([&](int n) { return make_float2(__ldg(a + n), has_b ? __ldg(b + n) : 0.f); }, buf,
                               1, lane, s_tw, active);
    if (active) {
      float2* oa = out + ra * out_pitch;
      float2* ob = out + rb * out_pitch;
      for (int k = lane; k <= L / 2; k += P) {
        const float2 zk = buf[lpos<PAD>(k)], zm = buf[lpos<PAD>((L - k) % L)];
        oa[k] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        if (has_b) ob[k] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
      }
    }
    __syncwarp();
  }
}

// ----------------------------------------------------------------- rows, C2R
// complex rows of length L/2+1 -> real rows of length L (unnormalised inverse).
// The imaginary parts of the k = 0 and k = L/2 terms are ignored (real-part
// semantics of a Hermitian inverse).
template <int L, int P>
__global__ void __launch_bounds__(256) k_rows_c2r(const float2* __restrict__ in, long in_pitch,
                                                  float* __restrict__ out, long out_pitch, long nrows,
                                                  const float2* __restrict__ g_tw) {
  constexpr int TEAMS = rows_teams(L, P);
  constexpr int PAD = line_pad(L);
  __shared__ float2 s_tw[L];
  __shared__ float2 s_line[TEAMS][row_line_len(L)];
  load_twiddles<L>(s_tw, g_tw);
  __syncthreads();
  const int team = threadIdx.x / P, lane = threadIdx.x % P;
  const long npairs = (nrows + 1) / 2;
  for (long pair0 = (long)blockIdx.x * TEAMS; pair0 < npairs; pair0 += (long)gridDim.x * TEAMS) {
    const long pair = pair0 + team;
    const bool active = pair < npairs;
    const long ra = 2 * pair, rb = 2 * pair + 1;
    const bool has_b = rb < nrows;
    float2* buf = s_line[team];
    const float2* a = in + ra * in_pitch;
    const float2* b = in + rb * in_pitch;
    // Hermitian extension of rows a and b packed as a + i b
    fft_line_in<L, 1, P, PAD>(
        [&](int n) {
          const bool lower = n <= L / 2;
          const int k = lower ? n : L - n;
          float2 A = a[k];
          float2 B = has_b ? b[k] : make_float2(0.f, 0.f);
          if (k == 0 || 2 * k == L) { A.y = 0.f; B.y = 0.f; }
          if (!lower) { A.y = -A.y; B.y = -B.y; }
          return make_float2(A.x - B.y, A.y + B.x);
        },
        buf, 1, lane, s_tw, active);
    if (active) {
      float* oa = out + ra * out_pitch;
      float* ob = out + rb * out_pitch;
      for (int n = lane; n < L; n += P) {
        const float2 z = buf[lpos<PAD>(n)];
        oa[n] = z.x;
        if (has_b) ob[n] = z.y;
      }
    }
    __syncwarp();
  }
}

// Whether a launch with this much dynamic shared memory needs the opt-in attribute: the 48 KiB that a
// kernel has without it also hold what the kernel declares statically (at most 1 KiB here; 360-point
// lines take 48,960 dynamic bytes, and with 256 static ones their launch was refused).
constexpr bool needs_smem_opt_in(size_t dynamic) { return dynamic + 1024 > 48 * 1024; }

// ----------------------------------------------------------------- strided columns
// Complex lines along a strided axis: element n of line (o, i) lives at
// base + o*outer_pitch + i + n*stride, for i in [0, inner), o in [0, outer); in == out is allowed
// (so neither pointer is restricted): a line's loads all precede its stores, by a barrier or, in
// single-stage plans, in one thread.
// A CTA transforms T consecutive lines (of the flattened (o, i), so that an inner extent that is no
// multiple of T leaves no partial tiles) with J threads each, threads of a half-warp on consecutive
// lines: the first stage takes its inputs from global memory, the last one stores its outputs there,
// and only the exchanges between stages cross shared memory, in place and without bank conflicts
// (twice per exchange; a tile copied in and out around teams that transform a line each crossed it
// eight times at 512 points).  Several CTAs per SM overlap one's loads with the others' stages.
template <int L>
struct ColsCfg {
  static constexpr int T = L <= 128 ? 32 : 16;
  static constexpr int MOST = 512 / T;
  // Threads per line: the count up to MOST whose rounds waste least over all stages, the largest such
  // (an even count, so that T J is a multiple of 32).
  static constexpr int padded_work(int J, int s = 0) {
    return radix_of(L, s) <= 1 ? 0
                               : (L / radix_of(L, s) + J - 1) / J * J * radix_of(L, s) + padded_work(J, s + 1);
  }
  static constexpr int best(int J, int found) {
    return J > MOST || J > 2 * min_butterflies(L) ? found
           : best(J + 2, padded_work(J) * 20 <= padded_work(found) * 21 ? J : found);
  }
  static constexpr int J = best(MOST / 4 + MOST / 4 % 2 > 2 ? MOST / 4 + MOST / 4 % 2 : 2,
                                MOST / 4 + MOST / 4 % 2 > 2 ? MOST / 4 + MOST / 4 % 2 : 2);
  static constexpr size_t smem = sizeof(float2) * (L + (size_t)L * T);
  static constexpr bool opt_in = needs_smem_opt_in(smem);
  static constexpr int by_smem = (int)((220 * 1024) / (smem + 1024));
  static constexpr int by_regs = 1024 / (T * J) > 1 ? 1024 / (T * J) : 1;  // 64 registers a thread
  static constexpr int min_blocks = by_smem < by_regs ? by_smem : by_regs;
};

// One stage of a tile's lines.  ld(n) / st(k, v): global element access of this thread's line.
template <int L, int SIGN, int T, int J, int S, class Ld, class St>
__device__ __forceinline__ void cols_stage(float2* line, int jt, bool active, const float2* tw, const Ld& ld,
                                           const St& st) {
  using I = InPlace<L, S>;
  constexpr bool FIRST = S == 0, LAST = S == n_stages(L) - 1;
#pragma unroll(FIRST ? 2 : 1)
  for (int b = jt; b < I::NB; b += J) {
    const int base = I::base(b), k = I::index(b);
    float2 v[I::R];
    if (FIRST) {
#pragma unroll
      for (int r = 0; r < I::R; ++r) v[r] = active ? ld(base + r * I::M) : make_float2(0.f, 0.f);
    } else {
#pragma unroll
      for (int r = 0; r < I::R; ++r) v[r] = line[(base + r * I::M) * T];
    }
    I::template run<SIGN>(v, k, tw);
    if (LAST) {
      if (active) {
#pragma unroll
        for (int r = 0; r < I::R; ++r) st(k + I::NS * r, v[r]);
      }
    } else {
#pragma unroll
      for (int r = 0; r < I::R; ++r) line[(base + r * I::M) * T] = v[r];
    }
  }
  if constexpr (!LAST) {
    __syncthreads();
    cols_stage<L, SIGN, T, J, S + 1>(line, jt, active, tw, ld, st);
  }
}

template <int L, int SIGN>
__global__ void __launch_bounds__(ColsCfg<L>::T * ColsCfg<L>::J, ColsCfg<L>::min_blocks) k_cols(
    const float2* in, float2* out, long stride, long inner, long lines, long outer_pitch,
    const float2* __restrict__ g_tw) {
  using C = ColsCfg<L>;
  extern __shared__ float2 smem[];
  float2* s_tw = smem;
  load_twiddles<L>(s_tw, g_tw);
  const int t = threadIdx.x % C::T, jt = threadIdx.x / C::T;
  const long c0 = (long)blockIdx.x * C::T;
  long o = c0 / inner, i = c0 - o * inner + t;  // the division is the same for the whole CTA
  while (i >= inner) {
    i -= inner;
    ++o;
  }
  const bool active = c0 + t < lines;
  const long at = o * outer_pitch + i;
  const float2* src = in + at;
  float2* dst = out + at;
  if constexpr (n_stages(L) > 1) __syncthreads();  // the twiddles
  cols_stage<L, SIGN, C::T, C::J, 0>(
      smem + L + t, jt, active, s_tw, [&](int n) { return src[(long)n * stride]; },
      [&](int k, float2 v) { dst[(long)k * stride] = v; });
}

// The forward z transform of `count` n^3 half spectra in place, with the weighting that follows it in a
// particle spectrum: q <- w b F, q(0) = 0, and the energies sum |q|^2 over the full spectra added in FP64
// (wgt: one half spectrum per volume, bp: one shared, either may be null).  The last stage's outputs are
// weighted in registers, so the spectra are not read and written once more.  Tiles stay inside a
// volume (blockIdx.y).
template <int L>
__global__ void __launch_bounds__(ColsCfg<L>::T * ColsCfg<L>::J, ColsCfg<L>::min_blocks) k_cols_weighted(
    float2* __restrict__ q, const float* __restrict__ wgt, const float* __restrict__ bp, double* __restrict__ energy,
    const float2* __restrict__ g_tw) {
  using C = ColsCfg<L>;
  constexpr int NH = L / 2 + 1, INNER = NH * L;
  constexpr int NT = C::T * C::J;
  static_assert(NT % 32 == 0, "whole warps");
  extern __shared__ float2 smem[];
  __shared__ double red[32];
  float2* s_tw = smem;
  load_twiddles<L>(s_tw, g_tw);
  const int t = threadIdx.x % C::T, jt = threadIdx.x / C::T;
  const int i = blockIdx.x * C::T + t;
  const bool active = i < INNER;
  const int kx = i % NH;
  const double hw = kx == 0 || 2 * kx == L ? 1.0 : 2.0;
  float2* line = q + (long)blockIdx.y * L * INNER + i;
  const float* wl = wgt ? wgt + (long)blockIdx.y * L * INNER + i : nullptr;
  const float* bl = bp ? bp + i : nullptr;
  double e = 0.0;
  if constexpr (n_stages(L) > 1) __syncthreads();  // the twiddles
  cols_stage<L, -1, C::T, C::J, 0>(
      smem + L + t, jt, active, s_tw, [&](int n) { return line[(long)n * INNER]; },
      [&](int k, float2 v) {
        float f = 1.f;
        if (wl) f *= __ldg(wl + (long)k * INNER);
        if (bl) f *= __ldg(bl + (long)k * INNER);
        if (i == 0 && k == 0) f = 0.f;
        v.x *= f;
        v.y *= f;
        line[(long)k * INNER] = v;
        e += (double)v.x * v.x + (double)v.y * v.y;
      });
  e *= hw;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int w = 0; w < NT / 32; ++w) tot += red[w];
    atomicAdd(energy + blockIdx.y, tot);
  }
}

// Host launchers (defined in fft_passes.cu); return EMC_OK or an error status.
emc_status launch_rows_r2c(int L, const float* in, long in_pitch, float2* out, long out_pitch, long nrows,
                           cudaStream_t st);
emc_status launch_rows_c2r(int L, const float2* in, long in_pitch, float* out, long out_pitch, long nrows,
                           cudaStream_t st);
emc_status launch_cols(int L, int sign, const float2* in, float2* out, long stride, long inner, long outer,
                       long outer_pitch, cudaStream_t st);

// Particle spectra: the R2C transform of `count` n^3 volumes, weighted, and their energies (cleared here);
// see k_cols_weighted.
emc_status weighted_spectra(const float* in, float2* out, int n, int count, const float* wgt, const float* bp,
                            double* energy, cudaStream_t st);

// Full 3-D R2C / C2R over a batch of volumes (x fastest).  c2r uses `scratch`
// ((nx/2+1)*ny*nz*batch float2) so that `in` is left untouched.
emc_status fft3_r2c(const float* in, float2* out, int nx, int ny, int nz, int batch, cudaStream_t st);
emc_status fft3_c2r(const float2* in, float* out, float2* scratch, int nx, int ny, int nz, int batch,
                    cudaStream_t st);

}  // namespace emc
