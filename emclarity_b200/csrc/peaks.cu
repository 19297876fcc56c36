// peaks.cu -- template-search post-processing: greedy peak picking with rotated erase masks,
// and the local normalisation of the pre-processing.
//
// Peak picking (alignment/BH_templateSearch3d_2.m:1100-1275, nPeaks = 1): repeat
//   [MAX, coord] = max(mag(:))                    (first index among ties)
//   if Ang(coord) > 0: record samplingRate * (c + centre of mass of mag in the 3^3 box - rmDim),
//     ANGLE_LIST(Ang(coord), :) and MAX; rotate the removal mask by the peak's Euler angles
//     (interpolator 'forward', C1) and zero mag in the (2 rmDim + 1)^3 box where it is >= cutoff
//   else: mag(coord) = 0
// while n <= maxPeaks, tries < maxTries and MAX > highThr.
// B200 layout: the map stays in HBM; a per-tile (8^3) maximum key (ordered value << 32 | ~index,
// so ties keep the first index) is kept up to date, and each step reduces only the tile keys,
// then rewrites only the tiles the erase box touched.  Steps run in batches of device launches
// that stop by themselves once the loop condition fails (a device status word), so the host
// synchronises once per batch, not once per peak.
//
// Local normalisation (BH_templateSearch3d_2.m:558-561, statistics/BH_movingAverage_2.m):
// mean = Gaussian-weighted moving average (kernel length = feature size, sigma 3, centred on
// (L - 1) / 2, normalised; EMC_gaussianKernel + EMC_convn 'same' after symmetric padding by
// ceil(L / 2)), rms = sqrt(mean(x^2) - mean(x)^2), x <- (x - mean) / rms.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "interp.cuh"

namespace emc {
namespace {

constexpr int kTile = 8;

__device__ __forceinline__ unsigned long long peak_key(float v, unsigned lin) {
  const unsigned u = __float_as_uint(v);
  const unsigned k = (v != v) ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));  // NaN never wins
  return ((unsigned long long)k << 32) | (0xffffffffu - lin);
}
__device__ __forceinline__ float key_value(unsigned long long key) {
  const unsigned k = (unsigned)(key >> 32);
  const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

struct PeakGeom {
  int nx, ny, nz;
  int tx, ty, tz;  // tiles per axis
  int rm;          // rmDim
  float cutoff;
  float sampling;
  float high_thr;
  int max_peaks, max_tries;
};

// Device state of the loop.
struct PeakState {
  int n_found;      // peaks recorded
  int tries;        // loop iterations
  int done;         // 1 once the loop condition failed
  int erase;        // 1: the last step recorded a peak and its box must be erased
  int cx, cy, cz;   // 0-based centre of the last step
  int angle;        // 1-based angle index of the last peak
  int reset_tile;   // tile to rescan after a single-voxel zeroing (-1 none)
  int pad;
};

// Maximum key of tile t.
__device__ unsigned long long tile_max(const float* mag, const PeakGeom& g, int t, int lane, int width) {
  const int tx = t % g.tx, ty = (t / g.tx) % g.ty, tz = t / (g.tx * g.ty);
  unsigned long long best = 0ull;
  for (int i = lane; i < kTile * kTile * kTile; i += width) {
    const int x = tx * kTile + (i & 7), y = ty * kTile + ((i >> 3) & 7), z = tz * kTile + (i >> 6);
    if (x < g.nx && y < g.ny && z < g.nz) {
      const unsigned lin = (unsigned)(((long)z * g.ny + y) * g.nx + x);
      const unsigned long long k = peak_key(mag[lin], lin);
      best = k > best ? k : best;
    }
  }
  return best;
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}

// One warp per tile.
__global__ void k_tile_keys(const float* __restrict__ mag, PeakGeom g, unsigned long long* __restrict__ keys) {
  const int warps = blockDim.x >> 5;
  const long ntiles = (long)g.tx * g.ty * g.tz;
  for (long t = blockIdx.x * (long)warps + (threadIdx.x >> 5); t < ntiles; t += (long)gridDim.x * warps) {
    const unsigned long long k = warp_max(tile_max(mag, g, (int)t, threadIdx.x & 31, 32));
    if ((threadIdx.x & 31) == 0) keys[t] = k;
  }
}

// One step of the loop, one CTA: global max over the tile keys, the decision, the centre of mass
// and the record.
__global__ void __launch_bounds__(1024) k_peak_select(float* __restrict__ mag, const float* __restrict__ ang,
                                                      PeakGeom g, const unsigned long long* __restrict__ keys,
                                                      const double* __restrict__ angle_list, int n_angles,
                                                      PeakState* __restrict__ st, double* __restrict__ peaks) {
  __shared__ unsigned long long red[32];
  __shared__ int s_done;
  if (threadIdx.x == 0) s_done = st->done;
  __syncthreads();
  if (s_done) return;
  const long ntiles = (long)g.tx * g.ty * g.tz;
  unsigned long long best = 0ull;
  for (long t = threadIdx.x; t < ntiles; t += blockDim.x) best = keys[t] > best ? keys[t] : best;
  best = warp_max(best);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) best = red[w] > best ? red[w] : best;
  red[0] = best;
  PeakState s = *st;
  s.erase = 0;
  s.reset_tile = -1;
  const float mx = key_value(best);
  // while n <= maxPeaks && tries < maxTries && MAX > highThr
  if (!(s.n_found < g.max_peaks && s.tries < g.max_tries && best != 0ull && mx > g.high_thr)) {
    s.done = 1;
    *st = s;
    return;
  }
  s.tries += 1;
  const unsigned lin = 0xffffffffu - (unsigned)(best & 0xffffffffu);
  const int x = (int)(lin % (unsigned)g.nx), y = (int)((lin / (unsigned)g.nx) % (unsigned)g.ny),
            z = (int)(lin / ((unsigned)g.nx * (unsigned)g.ny));
  const float a = ang[lin];
  if (a > 0.f) {
    // centre of mass of mag in the 3^3 box around the peak (bDist = 1 + round(log(1)) = 1)
    double sw = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
          const int xx = x + dx, yy = y + dy, zz = z + dz;
          if (xx < 0 || yy < 0 || zz < 0 || xx >= g.nx || yy >= g.ny || zz >= g.nz) continue;
          const double v = mag[((long)zz * g.ny + yy) * g.nx + xx];
          sw += v;
          sx += v * dx;
          sy += v * dy;
          sz += v * dz;
        }
    const int ai = (int)a;  // 1-based
    double* row = peaks + 10 * (size_t)s.n_found;
    // (c + cMass - rmDim) with c 1-based
    row[0] = g.sampling * ((x + 1) + sx / sw - g.rm);
    row[1] = g.sampling * ((y + 1) + sy / sw - g.rm);
    row[2] = g.sampling * ((z + 1) + sz / sw - g.rm);
    const bool in_list = ai >= 1 && ai <= n_angles;
    for (int k = 0; k < 3; ++k) row[3 + k] = in_list ? angle_list[3 * (size_t)(ai - 1) + k] : 0.0;
    row[6] = row[7] = row[8] = 0.0;
    row[9] = mx;
    s.n_found += 1;
    s.erase = 1;
    s.cx = x;
    s.cy = y;
    s.cz = z;
    s.angle = in_list ? ai : 0;
  } else {
    mag[lin] = 0.f;
    s.reset_tile = (z / kTile * g.ty + y / kTile) * g.tx + x / kTile;
  }
  *st = s;
}

// Zeroes mag in the (2 rm + 1)^3 box where the rotated removal mask is >= cutoff.  rmats: the
// sampling matrix (rows) of every angle, defineMatrix(angles, 'Bah', 'forward').
__global__ void k_peak_erase(float* __restrict__ mag, PeakGeom g, const PeakState* __restrict__ st,
                             const float* __restrict__ removal, const float* __restrict__ rmats) {
  const PeakState s = *st;
  if (!s.erase || s.done) return;
  const int r = 2 * g.rm + 1;
  const long nbox = (long)r * r * r;
  const float* m = rmats + 9 * (size_t)(s.angle > 0 ? s.angle - 1 : 0);
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nbox; i += (long)gridDim.x * blockDim.x) {
    const int bx = (int)(i % r), by = (int)((i / r) % r), bz = (int)(i / ((long)r * r));
    const int x = s.cx - g.rm + bx, y = s.cy - g.rm + by, z = s.cz - g.rm + bz;
    if (x < 0 || y < 0 || z < 0 || x >= g.nx || y >= g.ny || z >= g.nz) continue;
    // 'forward' with zero shift: s = R (p - c) + c, c = floor(r / 2) = rm, zero border
    const float u = (float)(bx - g.rm), v = (float)(by - g.rm), w = (float)(bz - g.rm);
    float rm_val = 1.f;  // no angle: erase the whole box
    if (s.angle > 0) {
      const float sx = fmaf(m[0], u, fmaf(m[1], v, m[2] * w)) + (float)g.rm;
      const float sy = fmaf(m[3], u, fmaf(m[4], v, m[5] * w)) + (float)g.rm;
      const float sz = fmaf(m[6], u, fmaf(m[7], v, m[8] * w)) + (float)g.rm;
      rm_val = sample_linear_border(removal, r, r, r, sx, sy, sz);
    }
    if (!(rm_val < g.cutoff)) mag[((long)z * g.ny + y) * g.nx + x] = 0.f;
  }
}

// Rescans the tiles the last step changed.
__global__ void k_peak_retile(const float* __restrict__ mag, PeakGeom g, const PeakState* __restrict__ st,
                              unsigned long long* __restrict__ keys) {
  const PeakState s = *st;
  const int warps = blockDim.x >> 5;
  const int wid = blockIdx.x * warps + (threadIdx.x >> 5);
  if (s.reset_tile >= 0) {
    if (wid == 0) {
      const unsigned long long k = warp_max(tile_max(mag, g, s.reset_tile, threadIdx.x & 31, 32));
      if ((threadIdx.x & 31) == 0) keys[s.reset_tile] = k;
    }
    return;
  }
  if (!s.erase) return;
  const int x0 = max(0, s.cx - g.rm) / kTile, x1 = min(g.nx - 1, s.cx + g.rm) / kTile;
  const int y0 = max(0, s.cy - g.rm) / kTile, y1 = min(g.ny - 1, s.cy + g.rm) / kTile;
  const int z0 = max(0, s.cz - g.rm) / kTile, z1 = min(g.nz - 1, s.cz + g.rm) / kTile;
  const int nx = x1 - x0 + 1, ny = y1 - y0 + 1, nt = nx * ny * (z1 - z0 + 1);
  for (int j = wid; j < nt; j += gridDim.x * warps) {
    const int t = ((z0 + j / (nx * ny)) * g.ty + (y0 + (j / nx) % ny)) * g.tx + (x0 + j % nx);
    const unsigned long long k = warp_max(tile_max(mag, g, t, threadIdx.x & 31, 32));
    if ((threadIdx.x & 31) == 0) keys[t] = k;
  }
}

// ---------------------------------------------------------------- moving average
// One separable pass along `axis` with symmetric (mirror, edge repeated) boundaries:
// out[x] = sum_t w[t] in[reflect(x + h - t)], h = floor(L / 2), summed in ascending t.
__device__ __forceinline__ int reflect_index(int q, int len) {
  // symmetric padding (padarray 'symmetric'): -1 -> 0, -2 -> 1, len -> len-1, ...
  if (q < 0) q = -q - 1;
  if (q >= len) q = 2 * len - q - 1;
  return q < 0 ? 0 : (q >= len ? len - 1 : q);
}

// The taps, passed by value: a call needs no table on the device and no wait for its upload.
constexpr int kMavgTaps = 96;
struct MavgTaps {
  float w[kMavgTaps];
};

// The value that a pass carries per voxel: x alone (moving average), or (x, x^2) in one register
// pair, whose two sums one packed FP32 multiply-add advances together (each rounds as alone).
template <bool SQ>
struct Tap;
template <>
struct Tap<false> {
  using T = float;
  static __device__ __forceinline__ T make(float v) { return v; }
  static __device__ __forceinline__ T fma(T w, T v, T acc) { return fmaf(w, v, acc); }
  static __device__ __forceinline__ T twice(float w) { return w; }
};
template <>
struct Tap<true> {
  using T = unsigned long long;
  static __device__ __forceinline__ T make(float v) { return pack2(v, v * v); }
  static __device__ __forceinline__ T fma(T w, T v, T acc) { return ffma2(w, v, acc); }
  static __device__ __forceinline__ T twice(float w) { return pack2(w, w); }
};

// R neighbouring outputs of one line: out[r] = sum_t w[t] ld(r + L - 1 - t), t ascending (w as
// Tap::twice made it).  The R inputs of a step sit in registers; a step shifts them by one and takes
// one new input, so an output costs (R + L - 1) / R fetches instead of L, and the R fetches of a
// round of steps are all in flight before its arithmetic.
template <bool SQ, int R, class Ld>
__device__ __forceinline__ void mavg_run(const typename Tap<SQ>::T* __restrict__ w, int L, const Ld& ld,
                                         typename Tap<SQ>::T out[R]) {
  using K = Tap<SQ>;
  typename K::T win[R];  // win[(r - t) mod R] = input r + L - 1 - t
#pragma unroll
  for (int r = 0; r < R; ++r) {
    out[r] = 0;
    if (r > 0) win[r] = ld(r + L - 1);
  }
  int t0 = 0;
#pragma unroll 1
  for (; t0 + R <= L; t0 += R) {
    typename K::T next[R];
#pragma unroll
    for (int k = 0; k < R; ++k) next[k] = ld(L - 1 - t0 - k);
#pragma unroll
    for (int k = 0; k < R; ++k) {
      win[(R - k) % R] = next[k];
      const typename K::T wt = w[t0 + k];
#pragma unroll
      for (int r = 0; r < R; ++r) out[r] = K::fma(wt, win[(r + R - k) % R], out[r]);
    }
  }
#pragma unroll
  for (int k = 0; k < R - 1; ++k) {
    if (t0 + k < L) {  // the same for every thread
      win[(R - k) % R] = ld(L - 1 - t0 - k);
      const typename K::T wt = w[t0 + k];
#pragma unroll
      for (int r = 0; r < R; ++r) out[r] = K::fma(wt, win[(r + R - k) % R], out[r]);
    }
  }
}

// 512 x 512 x 256, 16 taps: the local normalisation takes 871 us instead of 8,601 (six one-axis launches
// that fetched every tap through L1 with a division per index, over 1 GiB of scratch): 521 us in
// the xy launches and 337 in z, both bound by instruction issue (about 60 % of the slots).
//
// x and y passes of one z plane: a CTA smooths a kMavgTile^2 tile of plane z0 + blockIdx.z into
// plane (z mod ring) of buf.  The tile and its halo are read once into shared memory (reflected
// there), the x pass leaves its rows in shared memory (odd pitch, lanes on consecutive rows: no
// bank conflicts), the y pass reads them with lanes along x.
constexpr int kMavgTile = 64;
constexpr int kMavgRun = 8;
__host__ __device__ constexpr int mavg_span(int L) { return kMavgTile + L - 1; }
__host__ __device__ constexpr int mavg_in_pitch(int L) { return mavg_span(L) | 1; }
template <bool SQ>
size_t mavg_xy_smem(int L) {
  const size_t in = (sizeof(float) * mavg_span(L) * mavg_in_pitch(L) + 15) / 16 * 16;
  return in + sizeof(typename Tap<SQ>::T) * (mavg_span(L) * (kMavgTile + 1) + kMavgTaps) + sizeof(int) * 2 * mavg_span(L);
}

template <bool SQ>
__global__ void __launch_bounds__(256) k_mavg_xy(const float* __restrict__ in, typename Tap<SQ>::T* __restrict__ buf,
                                                 int nx, int ny, int z0, int ring, const MavgTaps taps, int L) {
  using K = Tap<SQ>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int span = mavg_span(L), pitch = mavg_in_pitch(L), h = L / 2;
  float* s_in = reinterpret_cast<float*>(smem_raw);
  typename K::T* s_x = reinterpret_cast<typename K::T*>(smem_raw + (sizeof(float) * span * pitch + 15) / 16 * 16);
  typename K::T* s_w = s_x + (size_t)span * (kMavgTile + 1);
  int* s_y = reinterpret_cast<int*>(s_w + kMavgTaps);
  int* s_xc = s_y + span;
  const int x0 = blockIdx.x * kMavgTile, y0 = blockIdx.y * kMavgTile, z = z0 + blockIdx.z;
  for (int t = threadIdx.x; t < L; t += blockDim.x) s_w[t] = K::twice(taps.w[t]);
  // rows and columns of the tile that exist; nothing past them is computed
  const int tw = min(kMavgTile, nx - x0), th = min(kMavgTile, ny - y0);
  const int cols = tw + L - 1, rows = th + L - 1;
  const float* src = in + (long)z * ny * nx;
  // the reflected source row and column of every tile row and column, once per tile
  for (int r = threadIdx.x; r < rows; r += blockDim.x) s_y[r] = reflect_index(y0 + h - (L - 1) + r, ny);
  for (int c = threadIdx.x; c < cols; c += blockDim.x) s_xc[c] = reflect_index(x0 + h - (L - 1) + c, nx);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < rows; r += 8) {
    const float* line = src + (long)s_y[r] * nx;
    for (int c = lane; c < cols; c += 32) cp_async4(s_in + r * pitch + c, line + s_xc[c]);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int xsegs = (tw + kMavgRun - 1) / kMavgRun;
  for (int i = threadIdx.x; i < rows * xsegs; i += blockDim.x) {
    const int r = i % rows, c0 = (i / rows) * kMavgRun;
    const float* line = s_in + r * pitch;
    typename K::T out[kMavgRun];
    // (the last run of a narrow tile also reads columns that were not filled, inside the full tile's
    // row; only outputs that are not stored depend on them.  The same holds in y and z.)
    mavg_run<SQ, kMavgRun>(s_w, L, [&](int k) { return K::make(line[c0 + k]); }, out);
#pragma unroll
    for (int k = 0; k < kMavgRun; ++k)
      if (c0 + k < tw) s_x[r * (kMavgTile + 1) + c0 + k] = out[k];
  }
  __syncthreads();
  typename K::T* dst = buf + (long)(z % ring) * ny * nx;
  const int ysegs = (th + kMavgRun - 1) / kMavgRun;
  for (int i = threadIdx.x; i < ysegs * kMavgTile; i += blockDim.x) {
    const int c = i % kMavgTile, r0 = (i / kMavgTile) * kMavgRun;
    if (c >= tw) continue;
    typename K::T out[kMavgRun];
    mavg_run<SQ, kMavgRun>(s_w, L, [&](int k) { return s_x[(r0 + k) * (kMavgTile + 1) + c]; }, out);
#pragma unroll
    for (int k = 0; k < kMavgRun; ++k)
      if (r0 + k < th) dst[(long)(y0 + r0 + k) * nx + x0 + c] = out[k];
  }
}

// z pass of planes [z0, z1) from the ring of smoothed planes.  A CTA takes kMavgCols columns and
// kMavgZ outputs of each: their kMavgZ + L - 1 inputs are copied into shared memory at once, so a
// column crosses the L2 (kMavgZ + L - 1) / kMavgZ times, and its runs are formed from there.
// SQ: vol <- (vol - mean) / sqrt(mean(x^2) - mean^2); else vol <- mean.
constexpr int kMavgZ = 32;
constexpr int kMavgCols = 128;
template <bool SQ>
size_t mavg_z_smem(int L) {
  return sizeof(typename Tap<SQ>::T) * ((size_t)(kMavgZ + L - 1) * kMavgCols + kMavgTaps) +
         sizeof(long) * (kMavgZ + L - 1);
}

template <bool SQ>
__global__ void __launch_bounds__(2 * kMavgCols) k_mavg_z(const typename Tap<SQ>::T* __restrict__ buf,
                                                          float* __restrict__ vol, long plane, int nz, int z0, int z1,
                                                          int ring, const MavgTaps taps, int L) {
  using K = Tap<SQ>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typename K::T* s_in = reinterpret_cast<typename K::T*>(smem_raw);
  typename K::T* s_w = s_in + (size_t)(kMavgZ + L - 1) * kMavgCols;
  const int zb = z0 + blockIdx.y * kMavgZ, h = L / 2;
  const int nout = min(kMavgZ, z1 - zb), nin = nout + L - 1;
  const int c = threadIdx.x % kMavgCols, half = threadIdx.x / kMavgCols;
  const long i = blockIdx.x * (long)kMavgCols + c;
  const bool in = i < plane;
  for (int t = threadIdx.x; t < L; t += blockDim.x) s_w[t] = K::twice(taps.w[t]);
  long* s_off = reinterpret_cast<long*>(s_w + kMavgTaps);  // each input's plane in the ring
  for (int k = threadIdx.x; k < nin; k += blockDim.x)
    s_off[k] = (long)(reflect_index(zb + k + h - (L - 1), nz) % ring) * plane;
  __syncthreads();
  for (int k = half; k < nin && in; k += 2) {
    const typename K::T* src = buf + s_off[k] + i;
    if constexpr (SQ) cp_async8(s_in + k * kMavgCols + c, src);
    else cp_async4(s_in + k * kMavgCols + c, src);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (!in) return;
  for (int r0 = half * kMavgRun; r0 < nout; r0 += 2 * kMavgRun) {
    float* dst = vol + (long)(zb + r0) * plane + i;
    float x[kMavgRun];
    if constexpr (SQ) {
#pragma unroll
      for (int k = 0; k < kMavgRun; ++k) x[k] = r0 + k < nout ? dst[k * plane] : 0.f;
    }
    typename K::T out[kMavgRun];
    mavg_run<SQ, kMavgRun>(s_w, L, [&](int k) { return s_in[(r0 + k) * kMavgCols + c]; }, out);
#pragma unroll
    for (int k = 0; k < kMavgRun; ++k) {
      if (r0 + k >= nout) break;
      if constexpr (SQ) {
        const float2 m = unpack2(out[k]);
        const float a = m.x;
        const float rms = sqrtf(m.y - a * a);
        dst[k * plane] = (x[k] - a) / rms;
      } else {
        dst[k * plane] = out[k];
      }
    }
  }
}

// One pass for kernels of more than kMavgTaps taps (features beyond the tiles' shared memory).
__global__ void k_mavg_pass(const float* __restrict__ in, float* __restrict__ out, int nx, int ny, int nz, int axis,
                            const float* __restrict__ w, int L) {
  const long n = (long)nx * ny * nz;
  const int h = L / 2;
  const int len = axis == 0 ? nx : axis == 1 ? ny : nz;
  const long stride = axis == 0 ? 1 : axis == 1 ? nx : (long)nx * ny;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int pos = axis == 0 ? (int)(i % nx) : axis == 1 ? (int)((i / nx) % ny) : (int)(i / ((long)nx * ny));
    const long base = i - (long)pos * stride;
    float acc = 0.f;
    for (int t = 0; t < L; ++t)
      acc = fmaf(w[t], __ldg(in + base + (long)reflect_index(pos + h - t, len) * stride), acc);
    out[i] = acc;
  }
}

__global__ void k_square(const float* __restrict__ in, float* __restrict__ out, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    out[i] = in[i] * in[i];
}

__global__ void k_local_norm(float* __restrict__ x, const float* __restrict__ avg, const float* __restrict__ avg2,
                             long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float a = avg[i];
    const float rms = sqrtf(avg2[i] - a * a);
    x[i] = (x[i] - a) / rms;
  }
}

int grid1(long n) { return (int)std::max<long>(1, std::min<long>((n + 255) / 256, 8L * device_sm_count())); }

// The normalised kernel of EMC_gaussianKernel([1, L], 3) (masking/EMC_gaussianKernel.m), single precision,
// normalised again as BH_movingAverage_2 does.
std::vector<float> mavg_kernel(int L) {
  std::vector<float> w(L);
  float s = 0.f;
  for (int t = 0; t < L; ++t) {
    const float v = ((float)t - (float)(L - 1) / 2.f) / 3.f;
    w[t] = expf(-0.5f * v * v);
    s += w[t];
  }
  float s2 = 0.f;
  for (int t = 0; t < L; ++t) {
    w[t] /= s;
    s2 += w[t];
  }
  for (int t = 0; t < L; ++t) w[t] /= s2;
  return w;
}

// Whether the ring of tiled passes takes a feature size: its taps fit the kernel argument and the
// tile's halo shared memory, and the grids their limits.  Wider features use one launch per axis.
bool mavg_tiled(int nx, int ny, int nz, int L) {
  return L <= kMavgTaps && (ny + kMavgTile - 1) / kMavgTile < 65536 && nz < 65536 &&
         ((long)nx * ny + 255) / 256 < (1l << 31);
}

// The three passes over a volume through a ring of xy-smoothed planes: slabs of z planes are
// smoothed in x and y into the ring, then the outputs whose inputs are all there are formed along z.
// The ring holds a slab of 64 MiB (at least kMavgZ planes) and the L - 1 planes before it: for tomograms of
// 512 x 512 and features up to 29 it stays in the L2 (94 MiB at 16, 120 at 29), so that the smoothed planes
// do not pass through HBM, and the scratch grows with a plane's area but not with nz.  vol may be `in`: a
// slab's outputs end h planes below the planes that later slabs still read.
template <bool SQ>
emc_status mavg_ring(const float* in, float* vol, int nx, int ny, int nz, const std::vector<float>& w,
                     cudaStream_t st) {
  using T = typename Tap<SQ>::T;
  const int L = (int)w.size(), h = L / 2;
  const long plane = (long)nx * ny;
  MavgTaps taps;
  for (int t = 0; t < L; ++t) taps.w[t] = w[t];
  // planes per slab: 64 MiB of smoothed planes (half the L2), whole runs of the z pass, all of a small volume
  long slab = (64l << 20) / (plane * (long)sizeof(T));
  slab = std::max<long>(kMavgZ, slab / kMavgZ * kMavgZ);
  slab = std::min<long>(slab, nz);
  const int ring = (int)std::min<long>(nz, slab + L - 1);
  // the kernels' limits are those of the widest feature, not of this call's: threads with different
  // features share them, and a smaller limit set between would refuse another thread's launch
  const size_t smem = mavg_xy_smem<SQ>(L), smem_z = mavg_z_smem<SQ>(L);
  EMC_CUDA(cudaFuncSetAttribute(k_mavg_xy<SQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)mavg_xy_smem<SQ>(kMavgTaps)));
  EMC_CUDA(cudaFuncSetAttribute(k_mavg_z<SQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)mavg_z_smem<SQ>(kMavgTaps)));
  T* buf = nullptr;
  EMC_CUDA(cudaMallocAsync((void**)&buf, sizeof(T) * plane * ring, st));
  const dim3 tiles((nx + kMavgTile - 1) / kMavgTile, (ny + kMavgTile - 1) / kMavgTile);
  int done = 0;  // outputs formed so far
  for (int z0 = 0; z0 < nz; z0 += (int)slab) {
    const int z1 = std::min(nz, z0 + (int)slab);
    k_mavg_xy<SQ><<<dim3(tiles.x, tiles.y, z1 - z0), 256, smem, st>>>(in, buf, nx, ny, z0, ring, taps, L);
    const int upto = z1 == nz ? nz : z1 - h;
    if (upto <= done) continue;
    k_mavg_z<SQ><<<dim3((unsigned)((plane + kMavgCols - 1) / kMavgCols), (upto - done + kMavgZ - 1) / kMavgZ),
                   2 * kMavgCols, smem_z, st>>>(buf, vol, plane, nz, done, upto, ring, taps, L);
    done = upto;
  }
  const cudaError_t e = cudaGetLastError();
  cudaFreeAsync(buf, st);
  EMC_CUDA(e);
  return EMC_OK;
}

emc_status mavg(const float* in, float* out, float* tmp, int nx, int ny, int nz, const float* d_w, int L,
                cudaStream_t st) {
  const long n = (long)nx * ny * nz;
  k_mavg_pass<<<grid1(n), 256, 0, st>>>(in, out, nx, ny, nz, 0, d_w, L);
  k_mavg_pass<<<grid1(n), 256, 0, st>>>(out, tmp, nx, ny, nz, 1, d_w, L);
  k_mavg_pass<<<grid1(n), 256, 0, st>>>(tmp, out, nx, ny, nz, 2, d_w, L);
  EMC_LAUNCH_CHECK();
  return EMC_OK;
}

}  // namespace
}  // namespace emc

extern "C" {

emc_status emc_tsearch_peaks(float* d_mag, const float* d_ang, int nx, int ny, int nz, const float* h_removal,
                             int rm_dim, float mask_cutoff, const double* angle_list, int n_angles, int max_peaks,
                             int max_tries, float high_thr, float sampling, double* h_peaks, int* n_found,
                             void* stream) {
  EMC_CHECK_ARG(d_mag && d_ang && h_removal && angle_list && h_peaks && n_found, "emc_tsearch_peaks: null argument");
  EMC_CHECK_ARG(nx > 0 && ny > 0 && nz > 0 && (long)nx * ny * nz < 0xffffffffL, "emc_tsearch_peaks: bad size");
  EMC_CHECK_ARG(rm_dim >= 1 && rm_dim < 256, "emc_tsearch_peaks: rm_dim %d", rm_dim);
  EMC_CHECK_ARG(n_angles >= 1 && max_peaks >= 0 && max_tries >= 0, "emc_tsearch_peaks: bad counts");
  cudaStream_t st = emc::as_stream(stream);
  emc::PeakGeom g;
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.tx = (nx + emc::kTile - 1) / emc::kTile;
  g.ty = (ny + emc::kTile - 1) / emc::kTile;
  g.tz = (nz + emc::kTile - 1) / emc::kTile;
  g.rm = rm_dim;
  g.cutoff = mask_cutoff;
  g.sampling = sampling;
  g.high_thr = high_thr;
  g.max_peaks = max_peaks;
  g.max_tries = max_tries;
  const long ntiles = (long)g.tx * g.ty * g.tz;
  const int r = 2 * rm_dim + 1;
  // forward sampling matrices of every angle (rows), defineMatrix(angles, 'Bah', 'forward')
  std::vector<float> mats(9 * (size_t)n_angles);
  for (int a = 0; a < n_angles; ++a) {
    double R[9];
    EMC_TRY(emc_define_matrix(angle_list + 3 * (size_t)a, 0, R));
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) mats[9 * (size_t)a + 3 * i + j] = (float)R[i + 3 * j];
  }
  unsigned long long* keys = nullptr;
  emc::PeakState* d_st = nullptr;
  float *d_rm = nullptr, *d_mats = nullptr;
  double *d_list = nullptr, *d_peaks = nullptr;
  emc_status rs = EMC_OK;
  auto alloc = [&](void** p, size_t b) {
    if (rs == EMC_OK && cudaMalloc(p, std::max<size_t>(b, 8)) != cudaSuccess) {
      emc::set_error("emc_tsearch_peaks: cudaMalloc(%zu) failed", b);
      rs = EMC_E_OOM;
    }
  };
  alloc((void**)&keys, sizeof(unsigned long long) * ntiles);
  alloc((void**)&d_st, sizeof(emc::PeakState));
  alloc((void**)&d_rm, sizeof(float) * (size_t)r * r * r);
  alloc((void**)&d_mats, sizeof(float) * mats.size());
  alloc((void**)&d_list, sizeof(double) * 3 * (size_t)n_angles);
  alloc((void**)&d_peaks, sizeof(double) * 10 * (size_t)std::max(1, max_peaks));
  emc::PeakState s0;
  memset(&s0, 0, sizeof(s0));
  s0.reset_tile = -1;
  if (rs == EMC_OK &&
      (cudaMemcpyAsync(d_st, &s0, sizeof(s0), cudaMemcpyHostToDevice, st) != cudaSuccess ||
       cudaMemcpyAsync(d_rm, h_removal, sizeof(float) * (size_t)r * r * r, cudaMemcpyHostToDevice, st) != cudaSuccess ||
       cudaMemcpyAsync(d_mats, mats.data(), sizeof(float) * mats.size(), cudaMemcpyHostToDevice, st) != cudaSuccess ||
       cudaMemcpyAsync(d_list, angle_list, sizeof(double) * 3 * (size_t)n_angles, cudaMemcpyHostToDevice, st) !=
           cudaSuccess))
    rs = EMC_E_CUDA;
  if (rs == EMC_OK) {
    emc::k_tile_keys<<<emc::grid1(ntiles * 32), 256, 0, st>>>(d_mag, g, keys);
    if (cudaGetLastError() != cudaSuccess) rs = EMC_E_CUDA;
  }
  const int erase_blocks = (int)std::max<long>(1, std::min<long>(((long)r * r * r + 255) / 256, 256));
  emc::PeakState hs = s0;
  // batches of steps; each kernel returns at once after the loop condition failed
  constexpr int kBatch = 64;
  while (rs == EMC_OK && !hs.done) {
    for (int b = 0; b < kBatch && rs == EMC_OK; ++b) {
      emc::k_peak_select<<<1, 1024, 0, st>>>(d_mag, d_ang, g, keys, d_list, n_angles, d_st, d_peaks);
      emc::k_peak_erase<<<erase_blocks, 256, 0, st>>>(d_mag, g, d_st, d_rm, d_mats);
      emc::k_peak_retile<<<8, 256, 0, st>>>(d_mag, g, d_st, keys);
      if (cudaGetLastError() != cudaSuccess) rs = EMC_E_CUDA;
    }
    if (rs == EMC_OK && (cudaMemcpyAsync(&hs, d_st, sizeof(hs), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                         cudaStreamSynchronize(st) != cudaSuccess))
      rs = EMC_E_CUDA;
  }
  if (rs == EMC_OK && hs.n_found > 0 &&
      (cudaMemcpyAsync(h_peaks, d_peaks, sizeof(double) * 10 * (size_t)hs.n_found, cudaMemcpyDeviceToHost, st) !=
           cudaSuccess ||
       cudaStreamSynchronize(st) != cudaSuccess))
    rs = EMC_E_CUDA;
  if (rs == EMC_E_CUDA) emc::set_error("emc_tsearch_peaks: %s", cudaGetErrorString(cudaGetLastError()));
  *n_found = rs == EMC_OK ? hs.n_found : 0;
  cudaStreamSynchronize(st);
  cudaFree(keys);
  cudaFree(d_st);
  cudaFree(d_rm);
  cudaFree(d_mats);
  cudaFree(d_list);
  cudaFree(d_peaks);
  return rs;
}

emc_status emc_moving_average(const float* d_in, int nx, int ny, int nz, int feature_size, float* d_out,
                              void* stream) {
  EMC_CHECK_ARG(d_in && d_out && nx > 0 && ny > 0 && nz > 0, "emc_moving_average: bad argument");
  EMC_CHECK_ARG(feature_size >= 2 && feature_size <= 2 * std::min(nx, std::min(ny, nz)),
                "emc_moving_average: feature size %d", feature_size);
  cudaStream_t st = emc::as_stream(stream);
  const std::vector<float> w = emc::mavg_kernel(feature_size);
  if (emc::mavg_tiled(nx, ny, nz, feature_size)) return emc::mavg_ring<false>(d_in, d_out, nx, ny, nz, w, st);
  const long n = (long)nx * ny * nz;
  float *d_w = nullptr, *tmp = nullptr;
  EMC_CUDA(cudaMallocAsync((void**)&d_w, sizeof(float) * feature_size, st));
  emc_status rs = EMC_OK;
  if (cudaMallocAsync((void**)&tmp, sizeof(float) * n, st) != cudaSuccess) rs = EMC_E_OOM;
  if (rs == EMC_OK && cudaMemcpyAsync(d_w, w.data(), sizeof(float) * feature_size, cudaMemcpyHostToDevice, st) !=
                          cudaSuccess)
    rs = EMC_E_CUDA;
  if (rs == EMC_OK) rs = emc::mavg(d_in, d_out, tmp, nx, ny, nz, d_w, feature_size, st);
  if (rs == EMC_E_OOM) emc::set_error("emc_moving_average: scratch allocation failed");
  cudaStreamSynchronize(st);  // w (host) is read by the async copy
  cudaFreeAsync(tmp, st);
  cudaFreeAsync(d_w, st);
  return rs;
}

emc_status emc_local_normalize(float* d_vol, int nx, int ny, int nz, int feature_size, void* stream) {
  EMC_CHECK_ARG(d_vol && nx > 0 && ny > 0 && nz > 0, "emc_local_normalize: bad argument");
  EMC_CHECK_ARG(feature_size >= 2 && feature_size <= 2 * std::min(nx, std::min(ny, nz)),
                "emc_local_normalize: feature size %d", feature_size);
  cudaStream_t st = emc::as_stream(stream);
  const std::vector<float> w = emc::mavg_kernel(feature_size);
  if (emc::mavg_tiled(nx, ny, nz, feature_size)) return emc::mavg_ring<true>(d_vol, d_vol, nx, ny, nz, w, st);
  const long n = (long)nx * ny * nz;
  float *d_w = nullptr, *buf = nullptr;
  EMC_CUDA(cudaMallocAsync((void**)&d_w, sizeof(float) * feature_size, st));
  emc_status rs = EMC_OK;
  if (cudaMallocAsync((void**)&buf, sizeof(float) * 4 * n, st) != cudaSuccess) rs = EMC_E_OOM;
  if (rs == EMC_OK && cudaMemcpyAsync(d_w, w.data(), sizeof(float) * feature_size, cudaMemcpyHostToDevice, st) !=
                          cudaSuccess)
    rs = EMC_E_CUDA;
  if (rs == EMC_OK) {
    float *avg = buf, *avg2 = buf + n, *sq = buf + 2 * n, *tmp = buf + 3 * n;
    rs = emc::mavg(d_vol, avg, tmp, nx, ny, nz, d_w, feature_size, st);
    if (rs == EMC_OK) {
      emc::k_square<<<emc::grid1(n), 256, 0, st>>>(d_vol, sq, n);
      rs = emc::mavg(sq, avg2, tmp, nx, ny, nz, d_w, feature_size, st);
    }
    if (rs == EMC_OK) {
      emc::k_local_norm<<<emc::grid1(n), 256, 0, st>>>(d_vol, avg, avg2, n);
      if (cudaGetLastError() != cudaSuccess) rs = EMC_E_CUDA;
    }
  }
  if (rs == EMC_E_OOM) emc::set_error("emc_local_normalize: scratch allocation failed");
  cudaStreamSynchronize(st);
  cudaFreeAsync(buf, st);
  cudaFreeAsync(d_w, st);
  return rs;
}

}  // extern "C"
