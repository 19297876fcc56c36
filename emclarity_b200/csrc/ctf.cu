// ctf.cu -- 2-D CTF images (mexCTF replacement) and the 3-D CTF^2 sampling-function wedge
// (mexSF3D replacement).
//
// Reference: mexFiles/include/core_headers.cuh:40-81 (ctfParams), mexFiles/utils/ctf.cu:12-130
// (kernels), mexFiles/mexCTF.cu:6-121, mexFiles/mexSF3D.cu:24-302.  The reference builds the
// SF3D volume with one texture upload and one launch per tilt; here all tilt images are made
// by one launch and a second launch accumulates every tilt into each (x, y) column.
#include <math.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fft.cuh"

namespace emc {

struct CtfDev {
  float cs_term, df_term, amp_phase, df1, df2, ast;
};

// ctfParams(doHalfGrid, doSqCTF, pix, lambda, Cs, AC, df1, df2, ast) evaluated in float on the
// host like the reference's __host__ constructor (core_headers.cuh:63-75).
static CtfDev make_ctf(const emc_ctf_params& p) {
  const float PI = 3.14159265358979323f;
  CtfDev c;
  c.amp_phase = atanf(p.amp_contrast / sqrtf(1.0f - p.amp_contrast * p.amp_contrast));
  c.df1 = 0.5f * (p.defocus1 + p.defocus2);
  c.df2 = 0.5f * (p.defocus1 - p.defocus2);
  c.ast = p.astig_deg * PI / 180.0f - (PI * (float)lrintf(p.astig_deg / 180.0f));
  c.cs_term = PI * 0.5f * p.cs_mm * 1e7f * (p.wavelength * p.wavelength * p.wavelength);
  c.df_term = PI * p.wavelength;
  return c;
}

struct CtfGrid {
  int dx, ny;      // output width (nx/2+1 or nx) and height
  int ox, oy;      // origin used by the centred / wrapped coordinate mapping
  int half, centred, squared;
  float fvx, fvy;  // Fourier voxel size 1/(pix*nx), 1/(pix*ny)
};

__device__ __forceinline__ float ctf_eval(const CtfDev& c, const CtfGrid& g, int x0, int y0, int* xs) {
  int x = x0, y = y0;
  if (g.centred) {
    y -= g.oy;
    if (!g.half) x -= g.ox;
  } else {
    if (y > g.oy) y -= g.ny;
    if (!g.half && x > g.ox) x -= g.dx;
  }
  *xs = x;
  const float fy = (float)y * g.fvy;
  const float fx = (float)x * g.fvx;
  const float phi = atan2f(fy, fx);
  const float r2 = fx * fx + fy * fy;
  const float v = sinf(c.cs_term * (r2 * r2) - c.df_term * r2 * (c.df1 + c.df2 * cosf(2.0f * (phi - c.ast))) -
                       c.amp_phase);
  return g.squared ? v * v : v;
}

// plain (ctf.cu:12-66) and exposure-filtered (ctf.cu:68-130) CTF images
__global__ void k_ctf2d(const CtfDev c, const CtfGrid g, int use_exposure, float radial_weight, float exposure,
                        float* __restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= g.dx || y >= g.ny) return;
  int xs;
  float v = ctf_eval(c, g, x, y, &xs);
  if (use_exposure) {
    const float rw = radial_weight * (xs == 0 ? 0.2f : fabsf((float)xs));
    int ys = y;
    if (g.centred) ys -= g.oy; else if (ys > g.oy) ys -= g.ny;
    const float fx = (float)xs * g.fvx, fy = (float)ys * g.fvy;
    const float r2 = fx * fx + fy * fy;
    // Grant-Grigorieff critical exposure a*s^(2b)+c with a = 0.24499, b = -0.8325 (on s^2), c = 2.8141
    v *= rw * expf((-0.5f * exposure) / (0.24499f * powf(r2, -0.8325f) + 2.81410f));
  }
  out[(long)y * g.dx + x] = v;
}

// What a tilt's CTF image shares between the volumes of a batch (full grid, centred,
// exposure-filtered): an image value is sin(a - b (df1 + df2 c) - amp)^2 w with a, b, c and w below,
// only the defocus pair depends on the volume.  One entry per pixel, [tilt][x][y].
struct SfTilt {
  CtfDev c;          // df1, df2 unused
  CtfGrid g;
  float sinA, cosA;  // of -tilt
  float occ, expo;
};

__device__ __forceinline__ float4 sf_pixel(const SfTilt& t, int x, int y) {
  const int xs = x - t.g.ox, ys = y - t.g.oy;
  const float fy = (float)ys * t.g.fvy;
  const float fx = (float)xs * t.g.fvx;
  const float phi = atan2f(fy, fx);
  const float r2 = fx * fx + fy * fy;
  const float rw = t.occ * (xs == 0 ? 0.2f : fabsf((float)xs));
  float4 v;
  // (products rounded on their own, as when they pass through the table)
  v.x = __fmul_rn(t.c.cs_term, r2 * r2);
  v.y = __fmul_rn(t.c.df_term, r2);
  v.z = cosf(2.0f * (phi - t.c.ast));
  // Grant-Grigorieff critical exposure as in k_ctf2d
  v.w = __fmul_rn(rw, expf((-0.5f * t.expo) / (0.24499f * powf(r2, -0.8325f) + 2.81410f)));
  return v;
}

__global__ void k_sf3d_tables(const SfTilt* __restrict__ tilts, int nx, int ny, float4* __restrict__ tab) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= nx || y >= ny) return;
  const SfTilt t = tilts[blockIdx.z];
  tab[((long)blockIdx.z * nx + x) * ny + y] = sf_pixel(t, x, y);
}

// Volumes whose image values lie together: K = 4 (a 16-byte load serves four volumes), or 1 for a
// single volume.
template <int K>
struct SfVols;
template <>
struct SfVols<4> {
  using Px = float4;
  using W = unsigned long long;
  unsigned long long a = 0ull, b = 0ull;  // two volumes a register pair, +0
  static __device__ __forceinline__ W weight(float w) { return pack2(w, w); }
  // += w ((1 - f) p + f q), g = 1 - f
  __device__ __forceinline__ void add(const Px& p, const Px& q, W g, W f, W w) {
    a = ffma2(w, ffma2(f, pack2(q.x, q.y), fmul2(g, pack2(p.x, p.y))), a);
    b = ffma2(w, ffma2(f, pack2(q.z, q.w), fmul2(g, pack2(p.z, p.w))), b);
  }
  __device__ __forceinline__ float get(int v) const {
    const float2 t = unpack2(v < 2 ? a : b);
    return v & 1 ? t.y : t.x;
  }
  static __device__ __forceinline__ Px pixel(const float (&v)[4]) { return make_float4(v[0], v[1], v[2], v[3]); }
};
template <>
struct SfVols<1> {
  using Px = float;
  using W = float;
  float a = 0.f;
  static __device__ __forceinline__ W weight(float w) { return w; }
  __device__ __forceinline__ void add(Px p, Px q, W g, W f, W w) {
    a = __fmaf_rn(w, __fmaf_rn(f, q, __fmul_rn(g, p)), a);
  }
  __device__ __forceinline__ float get(int) const { return a; }
  static __device__ __forceinline__ Px pixel(const float (&v)[1]) { return v[0]; }
};

// The tilt images of `count` volumes, [group of K volumes][tilt][x][y][volume] and one column of zeros
// after each group (lanes along y, as k_sf3d_volumes reads them).  A thread keeps its pixel's table
// entry and walks the groups: the radius, the angle and the exposure filter, most of an image's
// arithmetic, are formed once per pixel instead of per volume.  Without a table (K = 1) it forms the entry
// itself, once per volume: the table would be four fifths of the scratch (one volume of 1024 x 1024 x 16:
// 4,146 -> 976 us without it, most of the difference mapping memory).
template <int K>
__global__ void __launch_bounds__(256) k_sf3d_images(const float4* __restrict__ tab, const SfTilt* __restrict__ tilts,
                                                     const float2* __restrict__ df, int ntilts, long npix, int ny,
                                                     int count, int squared, typename SfVols<K>::Px* __restrict__ imgs) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int t = blockIdx.y;
  if (i >= npix) return;
  const float4 v = K == 1 ? sf_pixel(tilts[t], (int)(i / ny), (int)(i % ny)) : tab[(long)t * npix + i];
  const float amp = tilts[t].c.amp_phase;
  const long ngroup = npix * ntilts + ny;
  for (int g = blockIdx.z; g * K < count; g += gridDim.z) {
    float val[K], none[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      val[k] = none[k] = 0.f;
      if (g * K + k < count) {
        const float2 d = __ldg(df + (long)(g * K + k) * ntilts + t);
        const float s = sinf(v.x - v.y * (d.x + d.y * v.z) - amp);
        val[k] = (squared ? s * s : s) * v.w;
      }
    }
    imgs[g * ngroup + t * npix + i] = SfVols<K>::pixel(val);
    if (t == 0 && i < ny) imgs[g * ngroup + ntilts * npix + i] = SfVols<K>::pixel(none);
  }
}

// sf3dKernel (mexSF3D.cu:24-78) summed over tilts: every voxel within 4 px of a tilted central
// plane receives the sampled CTF^2 image (zero border) times the cosine edge weight, tilts in order.
// The plane tilts about y and its image rows are the volume's rows, so which tilts reach a voxel, the
// two image columns they sample and their weights depend on (x, z) alone.  A warp takes one (x, z)
// with its lanes along y: it tests the tilts 32 at a time, lists the few that reach it in shared
// memory, and then adds the listed columns for K volumes at once, group after group -- one coalesced
// load per row brings the K volumes' values, columns outside the image are its zero column, each
// output voxel is written once (the summation over z per column read and wrote it once per tilt).
// 128 volumes of 64^3 x 41 tilts: 208 us, their images 50 us, the whole call 4,023 -> 379 us.  With an
// 8-byte load per volume and two rows, and an atomic per warp and volume for the minimum, the sums took
// 372 us and the call 553: 262,144 atomics per launch on some 64 neighbouring words were the bound.  What
// is left is the latency of the list, the loads and the barriers of short CTAs: one group per CTA takes
// 212 us, six 244.
// The block's minimum goes to min_key (an ordered key per volume) when given.
constexpr int kSfX = 8;       // x positions (warps) per CTA: a row of 8 floats is one 32-byte sector
constexpr int kSfList = 128;  // tilts listed at a time

// V: rows per lane, 32 apart (2, or 1 when there are no more than 32 rows).
template <int V, int K>
__global__ void __launch_bounds__(32 * kSfX, 3) k_sf3d_volumes(const typename SfVols<K>::Px* __restrict__ imgs,
                                                            const SfTilt* __restrict__ tilts, int ntilts, int count,
                                                            int nx, int ny, int nz, int zbase, float* __restrict__ out,
                                                            unsigned* __restrict__ min_key) {
  using S = SfVols<K>;
  __shared__ int2 s_col[kSfX][kSfList];    // the two image columns
  __shared__ float2 s_wt[kSfX][kSfList];   // (x fraction, edge weight)
  __shared__ float s_out[K][32 * V][kSfX + 1];
  __shared__ float s_low[K][kSfX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x = blockIdx.x * kSfX + warp, z = zbase + blockIdx.y;
  const long ngroup = (long)nx * ny * ntilts + ny;
  const float PI = 3.14159265358979323f;
  const float ssx = (nx % 2 == 0) ? 0.5f : 0.f, ssz = (nz % 2 == 0) ? 0.5f : 0.f;
  const float u = (float)x - (float)nx / 2.0f;
  const float w = (float)(z - nz / 2);
  const int none = ntilts * nx;  // the zero column
  // the tilts t0 .. t0 + kSfList - 1 that reach (x, z), in order; returns how many
  auto list = [&](int t0) {
    int n = 0;
    for (int tb = t0; tb < min(t0 + kSfList, ntilts); tb += 32) {
      const int t = tb + lane;
      bool hit = false;
      int2 col = make_int2(none, none);
      float2 wt = make_float2(0.f, 0.f);
      if (t < ntilts && x < nx) {
        const float sA = tilts[t].sinA, cA = tilts[t].cosA;
        const float tw = -u * sA + ssz + w * cA;
        hit = !(tw < -4.0f || tw > 4.0f);
        float tu = u * cA + w * sA + ssx;
        tu = tu / (float)nx + 0.5f;
        const float tx = tu * (float)nx - 0.5f;
        const float fx0 = floorf(tx);
        const int c0 = (int)fx0;
        wt = make_float2(tx - fx0, (0.5f + 0.5f * cosf(tw * (PI / 4.0f))) * 0.25f);
        const int base = t * nx;
        if (c0 >= 0 && c0 < nx) col.x = base + c0;
        if (c0 + 1 >= 0 && c0 + 1 < nx) col.y = base + c0 + 1;
      }
      const unsigned hits = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int at = n + __popc(hits & ((1u << lane) - 1u));
        s_col[warp][at] = col;
        s_wt[warp][at] = wt;
      }
      n += __popc(hits);
    }
    __syncwarp();
    return n;
  };
  const bool once = ntilts <= kSfList;  // one list serves every y and every group
  int n = once ? list(0) : 0;
  for (int g = blockIdx.z; g * K < count; g += gridDim.z) {
    const int p0 = g * K, nvol = min(K, count - p0);
    float low[K];
#pragma unroll
    for (int v = 0; v < K; ++v) low[v] = INFINITY;
    for (int y0 = 0; y0 < ny; y0 += 32 * V) {
      S acc[V];
      // (lanes past the last row repeat it; what they form is not stored)
      const typename S::Px* img[V];
#pragma unroll
      for (int q = 0; q < V; ++q) img[q] = imgs + g * ngroup + min(y0 + lane + 32 * q, ny - 1);
      for (int t0 = 0; t0 < ntilts; t0 += kSfList) {
        if (!once) {
          __syncwarp();  // every lane is done with the previous list
          n = list(t0);
        }
#pragma unroll 2
        for (int k = 0; k < n; ++k) {
          const int2 col = s_col[warp][k];
          const float2 wt = s_wt[warp][k];
          const long oa = (long)col.x * ny, ob = (long)col.y * ny;
          typename S::Px a[V], b[V];
#pragma unroll
          for (int q = 0; q < V; ++q) {
            a[q] = __ldg(img[q] + oa);
            b[q] = __ldg(img[q] + ob);
          }
          const typename S::W wg = S::weight(1.f - wt.x), wf = S::weight(wt.x), we = S::weight(wt.y);
#pragma unroll
          for (int q = 0; q < V; ++q) acc[q].add(a[q], b[q], wg, wf, we);
        }
      }
#pragma unroll
      for (int q = 0; q < V; ++q)
#pragma unroll
        for (int v = 0; v < K; ++v) {
          const float val = acc[q].get(v);
          s_out[v][lane + 32 * q][warp] = val;
          if (x < nx && y0 + lane + 32 * q < ny) low[v] = fminf(low[v], val);  // NaN never becomes the minimum
        }
      __syncthreads();
      for (int i = threadIdx.x; i < nvol * 32 * V * kSfX; i += blockDim.x) {
        const int c = i % kSfX, r = (i / kSfX) % (32 * V), v = i / (kSfX * 32 * V);
        const int xo = blockIdx.x * kSfX + c, yo = y0 + r;
        if (xo < nx && yo < ny) out[(((long)(p0 + v) * nz + z) * ny + yo) * nx + xo] = s_out[v][r][c];
      }
      __syncthreads();
    }
    if (!min_key) continue;
    // one atomic per CTA and volume: the keys share a few sectors, whose atomics run one after another
#pragma unroll
    for (int v = 0; v < K; ++v) {
      float m = low[v];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) s_low[v][warp] = m;
    }
    __syncthreads();
    if (threadIdx.x < nvol) {
      float m = s_low[threadIdx.x][0];
#pragma unroll
      for (int q = 1; q < kSfX; ++q) m = fminf(m, s_low[threadIdx.x][q]);
      if (m < INFINITY) atomicMin(min_key + p0 + threadIdx.x, ordered_key(m));
    }
  }
}

// Binary Y-tilt-axis missing wedge of masking/BH_weightMask3d.m:103-120 on the half spectrum
// (FFT order, the ifftshift of the reference's centred grid), without the Gaussian smoothing
// (emc_binary_wedge applies it): theta = atan2d(kx, kz) is excluded inside the
// +/-(90 - tilt) cones around kz; the |kx|,|kz| <= 2 slab through the origin is kept; times the
// 'nyquist' radial window of BH_bandpass3d (:124-131 of BH_weightMask3d.m).  Optionally times the 3-D CTF of |k|
// (ctf.cu:45-62 with the radius taken in 3-D).
__global__ void k_wedge_ctf(int n, float max_cone, float min_cone, int use_ctf, int squared, const CtfDev c,
                            float inv_box_pix, float* __restrict__ out) {
  const int nh = n / 2 + 1;
  const long total = (long)nh * n * n;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    // signed frequencies of the ifftshifted centred grid: for even n the Nyquist index is -n/2
    const int kx0 = (int)(i % nh);
    const int ky0 = (int)((i / nh) % n), kz0 = (int)(i / ((long)nh * n));
    const int kx = 2 * kx0 < n ? kx0 : kx0 - n;
    const int ky = 2 * ky0 < n ? ky0 : ky0 - n;
    const int kz = 2 * kz0 < n ? kz0 : kz0 - n;
    const float theta = atan2f((float)kx, (float)kz) * (180.0f / 3.14159265358979323f);
    const bool excluded = (180.0f - min_cone <= theta || theta <= max_cone - 180.0f) ||
                          (-min_cone <= theta && theta <= max_cone);
    float w = excluded ? 0.f : 1.f;
    if (abs(kx) <= 2 && abs(kz) <= 2) w = 1.f;
    const float r2i = (float)(kx * kx + ky * ky + kz * kz);
    // BH_bandpass3d(size, 0, 0, 0, METHOD, 'nyquist'): 1 below 0.485 cycles/pixel, Gaussian
    // roll-off of width 1.5/n beyond (masking/BH_bandpass3d.m:60-77, :88-92)
    const float rn = sqrtf(r2i) / (float)n;
    if (rn >= 0.485f) {
      const float roll = 1.5f / (float)n;
      w *= expf(-(rn - 0.485f) * (rn - 0.485f) / (2.f * roll * roll));
    }
    if (use_ctf && w != 0.f) {
      const float r2 = r2i * inv_box_pix * inv_box_pix;
      const float v = sinf(c.cs_term * (r2 * r2) - c.df_term * r2 * c.df1 - c.amp_phase);
      w *= squared ? v * v : v;
    }
    out[i] = w;
  }
}

static CtfGrid make_grid(int nx, int ny, int half, int squared, int centred, float pix) {
  CtfGrid g;
  g.half = half;
  g.centred = centred;
  g.squared = squared;
  g.ny = ny;
  g.dx = half ? nx / 2 + 1 : nx;
  g.ox = half ? 0 : nx / 2;
  g.oy = ny / 2;
  g.fvx = 1.0f / (pix * (float)nx);
  g.fvy = 1.0f / (pix * (float)ny);
  return g;
}

// SF3D - (min(SF3D(:)) - 1e-4) (masking/BH_weightMaskMex.m:55) from the volume's ordered minimum key.
__global__ void k_vol_sub_min(float* __restrict__ v, long n, const unsigned* __restrict__ key, float eps) {
  float* dst = v + (long)blockIdx.y * n;
  const unsigned k = key[blockIdx.y];
  const unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  const float mn = __uint_as_float(u);
  const float off = mn - eps;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = dst[i] - off;
}

// SF3D volumes of a batch: tilts ts (shared), defocus pairs df [volume][tilt]; `shifted` subtracts
// min - 1e-4 from each.  Volumes go through in chunks whose tilt images (and so, at the usual 40
// tilts, volumes) stay in the L2 between the launches.  K: volumes per group.
template <int K>
static emc_status sf3d_batch(const std::vector<SfTilt>& ts, const std::vector<float2>& df, int count, int nx, int ny,
                             int nz, int squared, bool shifted, float* d_out, cudaStream_t st) {
  using Px = typename SfVols<K>::Px;
  const int n = (int)ts.size();
  const long npix = (long)nx * ny, nv = npix * nz;
  const size_t group = sizeof(Px) * ((size_t)n * npix + ny);  // bytes of a group's images
  const int ngroups = (count + K - 1) / K;
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>({(size_t)ngroups, (size_t)(48ull << 20) / group, 65535}));
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t t_bytes = up(sizeof(SfTilt) * n), d_bytes = up(sizeof(float2) * df.size());
  const size_t k_bytes = up(sizeof(unsigned) * count), tab_bytes = K == 1 ? 0 : up(sizeof(float4) * (size_t)n * npix);
  std::vector<char> host(t_bytes + d_bytes);
  memcpy(host.data(), ts.data(), sizeof(SfTilt) * n);
  memcpy(host.data() + t_bytes, df.data(), sizeof(float2) * df.size());
  char* buf = nullptr;
  EMC_CUDA(cudaMallocAsync(&buf, t_bytes + d_bytes + k_bytes + tab_bytes + group * chunk, st));
  const SfTilt* d_t = reinterpret_cast<const SfTilt*>(buf);
  const float2* d_df = reinterpret_cast<const float2*>(buf + t_bytes);
  unsigned* keys = reinterpret_cast<unsigned*>(buf + t_bytes + d_bytes);
  float4* tab = reinterpret_cast<float4*>(buf + t_bytes + d_bytes + k_bytes);
  Px* imgs = reinterpret_cast<Px*>(buf + t_bytes + d_bytes + k_bytes + tab_bytes);
  cudaError_t e = cudaMemcpyAsync(buf, host.data(), host.size(), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && shifted) e = cudaMemsetAsync(keys, 0xff, sizeof(unsigned) * count, st);
  if (e == cudaSuccess && K > 1) {
    k_sf3d_tables<<<dim3((ny + 31) / 32, (nx + 7) / 8, n), dim3(32, 8), 0, st>>>(d_t, nx, ny, tab);
    e = cudaGetLastError();
  }
  for (int g0 = 0; g0 < ngroups && e == cudaSuccess; g0 += chunk) {
    const int p0 = g0 * K, cnt = std::min(chunk * K, count - p0), gs = (cnt + K - 1) / K;
    float* out = d_out + (size_t)p0 * nv;
    // enough groups side by side to fill the chip when one group's pixels do not
    const unsigned blocks = (unsigned)((npix + 255) / 256);
    const unsigned zs = (unsigned)std::min<long>(gs, 1 + 16L * device_sm_count() / ((long)blocks * n));
    k_sf3d_images<K><<<dim3(blocks, n, zs), 256, 0, st>>>(tab, d_t, d_df + (size_t)p0 * n, n, npix, ny, cnt, squared, imgs);
    const unsigned gx = (nx + kSfX - 1) / kSfX;
    for (int z0 = 0; z0 < nz; z0 += 65535) {
      // a CTA's list serves as many groups as leave about eight waves of CTAs (two groups at 64 volumes of 64^3)
      const int gy = std::min(nz - z0, 65535);
      const long per = std::max<long>(1, std::min<long>(gs, (long)gx * gy * gs / (24L * device_sm_count())));
      (ny > 32 ? k_sf3d_volumes<2, K> : k_sf3d_volumes<1, K>)<<<dim3(gx, gy, (unsigned)((gs + per - 1) / per)),
                                                                 32 * kSfX, 0, st>>>(
          imgs, d_t, n, cnt, nx, ny, nz, z0, out, shifted ? keys + p0 : nullptr);
    }
    if (shifted) {
      const int gxm = (int)std::max<long>(1, std::min<long>((nv + 1023) / 1024, 64));
      for (int q = 0; q < cnt; q += 65535)
        k_vol_sub_min<<<dim3(gxm, std::min(cnt - q, 65535)), 256, 0, st>>>(out + (size_t)q * nv, nv, keys + p0 + q, 1e-4f);
    }
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFreeAsync(buf, st);
  EMC_CUDA(e);
  return EMC_OK;
}

}  // namespace emc

extern "C" {

emc_status emc_ctf2d(const emc_ctf_params* p, int nx, int ny, int half, int squared, int centred, float* d_out,
                     void* stream) {
  EMC_CHECK_ARG(p && d_out, "emc_ctf2d: null argument");
  EMC_CHECK_ARG(nx > 0 && ny > 0, "emc_ctf2d: bad size");
  EMC_CHECK_ARG(p->pixel_size > 0.f && p->amp_contrast >= 0.f && p->amp_contrast < 1.f, "emc_ctf2d: bad parameters");
  const emc::CtfDev c = emc::make_ctf(*p);
  const emc::CtfGrid g = emc::make_grid(nx, ny, half, squared, centred, p->pixel_size);
  dim3 block(32, 8), grid((g.dx + 31) / 32, (ny + 7) / 8);
  emc::k_ctf2d<<<grid, block, 0, emc::as_stream(stream)>>>(c, g, 0, 0.f, 0.f, d_out);
  EMC_LAUNCH_CHECK();
  return EMC_OK;
}

emc_status emc_ctf2d_exposure(const emc_ctf_params* p, int nx, int ny, int half, int squared, int centred,
                              float radial_weight, float total_exposure, float* d_out, void* stream) {
  EMC_CHECK_ARG(p && d_out, "emc_ctf2d_exposure: null argument");
  EMC_CHECK_ARG(nx > 0 && ny > 0, "emc_ctf2d_exposure: bad size");
  const emc::CtfDev c = emc::make_ctf(*p);
  const emc::CtfGrid g = emc::make_grid(nx, ny, half, squared, centred, p->pixel_size);
  dim3 block(32, 8), grid((g.dx + 31) / 32, (ny + 7) / 8);
  emc::k_ctf2d<<<grid, block, 0, emc::as_stream(stream)>>>(c, g, 1, radial_weight, total_exposure, d_out);
  EMC_LAUNCH_CHECK();
  return EMC_OK;
}

emc_status emc_wedge_ctf_weight(int n, float tilt_min_deg, float tilt_max_deg, const emc_ctf_params* ctf,
                                int squared, float* d_out, void* stream) {
  EMC_CHECK_ARG(d_out && n >= 2, "emc_wedge_ctf_weight: bad argument");
  EMC_CHECK_ARG(tilt_min_deg <= tilt_max_deg, "emc_wedge_ctf_weight: tilt_min > tilt_max");
  // maxTilt = 90 - |min(tilts)|, minTilt = 90 - |max(tilts)| (BH_weightMask3d.m:109-110)
  const float max_cone = 90.0f - fabsf(tilt_min_deg), min_cone = 90.0f - fabsf(tilt_max_deg);
  emc::CtfDev c{};
  float inv_box_pix = 0.f;
  if (ctf) {
    EMC_CHECK_ARG(ctf->pixel_size > 0.f, "emc_wedge_ctf_weight: pixel size");
    c = emc::make_ctf(*ctf);
    inv_box_pix = 1.0f / ((float)n * ctf->pixel_size);
  }
  const long total = (long)(n / 2 + 1) * n * n;
  const int blocks = (int)std::min<long>((total + 255) / 256, 4L * emc::device_sm_count());
  emc::k_wedge_ctf<<<blocks, 256, 0, emc::as_stream(stream)>>>(n, max_cone, min_cone, ctf ? 1 : 0, squared, c,
                                                                inv_box_pix, d_out);
  EMC_LAUNCH_CHECK();
  return EMC_OK;
}

emc_status emc_sf3d(int half, int squared, const unsigned size[3], const float* pix, const float* wavelength,
                    const float* cs_mm, const float* df1, const float* df2, const float* astig_deg,
                    const float* amp_contrast, unsigned n_tilts, const float* tilt_deg, const float* exposure,
                    const float* occupancy, float* d_out, void* stream) {
  EMC_CHECK_ARG(size && pix && wavelength && cs_mm && df1 && df2 && astig_deg && amp_contrast && tilt_deg &&
                    exposure && occupancy && d_out,
                "emc_sf3d: null argument");
  EMC_CHECK_ARG(half == 0, "emc_sf3d: only the full grid is built (as in the reference)");
  EMC_CHECK_ARG(n_tilts > 0 && n_tilts < 100000, "emc_sf3d: n_tilts %u", n_tilts);
  const int nx = (int)size[0], ny = (int)size[1], nz = (int)size[2];
  EMC_CHECK_ARG(nx > 0 && ny > 0 && nz > 0, "emc_sf3d: bad size");
  std::vector<emc::SfTilt> ts(n_tilts);
  std::vector<float2> df(n_tilts);
  for (unsigned t = 0; t < n_tilts; ++t) {
    emc_ctf_params p{pix[t], wavelength[t], cs_mm[t], amp_contrast[t], df1[t], df2[t], astig_deg[t]};
    ts[t].c = emc::make_ctf(p);
    df[t] = make_float2(ts[t].c.df1, ts[t].c.df2);
    ts[t].g = emc::make_grid(nx, ny, 0, squared, 1, pix[t]);
    // sincosf(deg_2_rad(-tilt)) (mexSF3D.cu:131-135)
    const float a = -tilt_deg[t] * 3.14159265358979323f / 180.0f;
    ts[t].sinA = sinf(a);
    ts[t].cosA = cosf(a);
    ts[t].occ = occupancy[t];
    ts[t].expo = exposure[t];
  }
  return emc::sf3d_batch<1>(ts, df, 1, nx, ny, nz, squared, false, d_out, emc::as_stream(stream));
}

// BH_weightMaskMex(SIZE, SAMPLING, TLT, xyzSubTomo, reconGeometry) for a batch of particles
// (masking/BH_weightMaskMex.m:1-60), arithmetic in single precision like the reference (TLT is cast to
// single first, :11).
emc_status emc_sf3d_particles(const unsigned size[3], double sampling, const double* tlt, int rows, int cols,
                              const double* xyz, const double recon_geometry[6], int count, float* d_out,
                              void* stream) {
  EMC_CHECK_ARG(size && tlt && xyz && recon_geometry && d_out, "emc_sf3d_particles: null argument");
  EMC_CHECK_ARG(rows > 0 && cols >= 19, "emc_sf3d_particles: tilt table %d x %d (needs 19 columns)", rows, cols);
  EMC_CHECK_ARG(count >= 0, "emc_sf3d_particles: count %d", count);
  if (count == 0) return EMC_OK;
  // sortrows(TLT, 1): stable ascending sort on column 1, then single precision
  std::vector<int> order(rows);
  for (int r = 0; r < rows; ++r) order[r] = r;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return tlt[(size_t)a * cols] < tlt[(size_t)b * cols]; });
  auto T = [&](int r, int c) { return (float)tlt[(size_t)order[r] * cols + (c - 1)]; };  // 1-based column
  const int n = rows;
  std::vector<float> pix(n), lam(n), cs(n), ac(n), def0(n), ddf(n), dphi(n), tilt(n), expo(n), occ(n);
  float dose_mean = 0.f;
  for (int r = 0; r < n; ++r) dose_mean += T(r, 14);
  dose_mean /= (float)n;
  std::vector<float> elastic(n);
  float el_max = 0.f;
  for (int r = 0; r < n; ++r) {
    pix[r] = T(r, 16) * (float)sampling * 1e10f;
    cs[r] = T(r, 17) * 1e3f;
    lam[r] = T(r, 18) * 1e10f;
    ac[r] = T(r, 19);
    def0[r] = -T(r, 15) * 1e10f;
    ddf[r] = T(r, 12) * 1e10f;
    dphi[r] = T(r, 13) * 180.0f / 3.14159265358979323846f;
    tilt[r] = T(r, 4);
    expo[r] = T(r, 11);
    // fractionOfElastics = exp(-thickness / (cosd(tilt) * 400)), thickness 75 nm, normalised (:44-46)
    elastic[r] = expf(-75.0f / (cosf(tilt[r] * 3.14159265358979323846f / 180.0f) * 400.0f));
    el_max = std::max(el_max, elastic[r]);
  }
  for (int r = 0; r < n; ++r) occ[r] = (elastic[r] / el_max) * (T(r, 14) / dose_mean);
  // originVol = ceil((reconGeometry(1, 1:3) + 1) / 2), reconShift = reconGeometry(2, :) (:17-20)
  double origin[3], rshift[3];
  for (int d = 0; d < 3; ++d) {
    origin[d] = ceil((recon_geometry[d] + 1.0) / 2.0);
    rshift[d] = recon_geometry[3 + d];
  }
  const int nx = (int)size[0], ny = (int)size[1], nz = (int)size[2];
  EMC_CHECK_ARG(nx > 0 && ny > 0 && nz > 0 && n < 65536, "emc_sf3d_particles: bad size or tilt count");
  std::vector<emc::SfTilt> ts(n);
  std::vector<float> sn(n), co(n);
  for (int r = 0; r < n; ++r) {
    const emc_ctf_params cp{pix[r], lam[r], cs[r], ac[r], 0.f, 0.f, dphi[r]};
    ts[r].c = emc::make_ctf(cp);
    ts[r].g = emc::make_grid(nx, ny, 0, 1, 1, pix[r]);
    const float a = -tilt[r] * 3.14159265358979323f / 180.0f;  // sincosf(deg_2_rad(-tilt)) (mexSF3D.cu:131-135)
    ts[r].sinA = sinf(a);
    ts[r].cosA = cosf(a);
    ts[r].occ = occ[r];
    ts[r].expo = expo[r];
    // rTilt = defineMatrix(tilt, 'TILT', 'forwardVector') = [c 0 s; 0 1 0; -s 0 c]; z of rTilt * v (:27-30)
    const float b = tilt[r] * (3.14159265358979323846f / 180.0f);
    sn[r] = sinf(b);
    co[r] = cosf(b);
  }
  // every (particle, tilt) defocus pair, offset by the particle's height along the beam
  std::vector<float2> df((size_t)count * n);
  for (int p = 0; p < count; ++p) {
    const float vx = (float)(xyz[3 * (size_t)p] - origin[0] + rshift[0]);
    const float vz = (float)(xyz[3 * (size_t)p + 2] - origin[2] + rshift[2]);
    for (int r = 0; r < n; ++r) {
      const float z = -sn[r] * vx + co[r] * vz;
      const float d = def0[r] - z * pix[r];
      const float d1 = d + ddf[r], d2 = d - ddf[r];
      df[(size_t)p * n + r] = make_float2(0.5f * (d1 + d2), 0.5f * (d1 - d2));
    }
  }
  // Groups of four share a table: 32 bytes of scratch per pixel and tilt.  Past 128 MiB of that (41 tilts
  // above 320^2) volumes go one at a time, with 4 bytes: mapping the scratch then costs more than the
  // groups save (41 tilts, two volumes of 800 x 800 x 4: 1,052 us against 3,984; three of 512 x 512 x 16: 823
  // against 1,860), and the call stays within the memory that it took without groups.
  const bool groups = count > 1 && 32 * (size_t)n * nx * ny <= (128ull << 20);
  return (groups ? emc::sf3d_batch<4> : emc::sf3d_batch<1>)(ts, df, count, nx, ny, nz, 1, true, d_out,
                                                            emc::as_stream(stream));
}

}  // extern "C"
