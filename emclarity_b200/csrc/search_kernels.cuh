// search_kernels.cuh -- the three fused passes of one CC evaluation (particle, orientation).
//
// Data flow per evaluation e (box n, half width nh = n/2+1, peak radius r, window w = 2r+1):
//   pass A  (CTA = z-planes, one gather r = mask .* I(M (p - c - t) + c) into registers
//            at a time)          (no weight on the reference: sums of r and r^2, the DC-free energy by
//                                Parseval), R2C along x (two rows per complex FFT), FFT along y,
//                                in place in one shared-memory plane
//                                -> S1[e][ky][z][column]                   (~n * n * nh c64)
//   pass B  (CTA = one ky row)   FFT along z, X = Q .* conj(wref .* R) .* wdgMask, X(0) = 0,
//                                E_R = sum |wref .* R .* wdgMask|^2 when either weight is set (both
//                                formed in registers between the transforms), inverse FFT along z,
//                                keep the w output planes |sz| <= r
//                                -> S2[e][j][ky][kx], planes in pass C's tile layout  (~w * n * nh c64)
//   pass C  (CTA = one sz plane) inverse FFT along y, C2R along x for the w rows |sy| <= r,
//                                normalise by sqrt(E_R E_P), spherical peak mask,
//                                argmax -> atomicMax on a 64-bit (cc, -index) key
// The reference computes the whole map (BH_multi_xcf_Translational_2.m:35-38) and then
// masks it (BH_multi_xcf_Translational.m:33-42); only the masked window is evaluated here.
#pragma once
#include "interp.cuh"

namespace emc {

struct DevParticle {
  const float2* spec;  // Q = refWdg .* P, [z][y][kx]
  const float* wedge;  // wdgMask, the weight on the rotated reference, [z][y][kx] or null (= 1)
  double energy;       // E_P = sum |Q|^2
  double prior[9];     // column-major
  float shift[3];
  int ref;
  int box;
  int orient_begin;
  long eval_base;      // index of this particle's first (p, o) pair in the output order
};

struct DevRef {
  const void* data;    // n^3, float or bf16
  const float* mask;   // n^3 or null
  const float* wref;   // nh*n*n or null
  int n;
  int dtype;
  const void* cells;   // (n+1)^3 trilinear corner cells (see build_cells) or null
  const unsigned* mask_rows;  // per (z, y) row: lo | hi << 16, the x extent [lo, hi) of mask != 0, or null
  const void* bricks;         // the corner cells in pass A's bricks (brick_index), or null
  const float* mask_tiles;    // the mask in pass A's tiles (mask_tile_index), or null
};

// Trilinear corner cells: cell (i, j, k), i, j, k in [-1, n-1], holds the 8 voxels
// v(i+a, j+b, k+c), a, b, c in {0, 1}, in the order (000, 100, 010, 110, 001, 101, 011, 111),
// zero outside the volume.  One 32-byte (FP32) or 16-byte (BF16) vector load fetches every
// corner a trilinear sample needs, instead of eight scattered 4-byte loads.
template <typename T>
struct CellT;
template <>
struct CellT<float> {
  float4 lo, hi;
};
template <>
struct CellT<__nv_bfloat16> {
  uint4 v;
};

__device__ __forceinline__ void cell_values(const CellT<float>& c, float v[8]) {
  v[0] = c.lo.x; v[1] = c.lo.y; v[2] = c.lo.z; v[3] = c.lo.w;
  v[4] = c.hi.x; v[5] = c.hi.y; v[6] = c.hi.z; v[7] = c.hi.w;
}
__device__ __forceinline__ void cell_values(const CellT<__nv_bfloat16>& c, float v[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&c.v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(p[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
// One 256-bit read-only load (sm_100) under a predicate: the whole 32-byte cell in a single request, so
// the cell's sector is looked up once instead of once per 16-byte half.  Cells are 32-byte aligned.  An
// inactive lane's value is undefined and its access is not made.
__device__ __forceinline__ CellT<float> load_cell_if(const CellT<float>* p, bool on) {
  CellT<float> c;
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %9, 0;\n"
      " @q ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n}\n"
      : "=f"(c.lo.x), "=f"(c.lo.y), "=f"(c.lo.z), "=f"(c.lo.w), "=f"(c.hi.x), "=f"(c.hi.y), "=f"(c.hi.z),
        "=f"(c.hi.w)
      : "l"(p), "r"((int)on));
  return c;
}
__device__ __forceinline__ CellT<__nv_bfloat16> load_cell_if(const CellT<__nv_bfloat16>* p, bool on) {
  CellT<__nv_bfloat16> c;
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %5, 0;\n @q ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n}\n"
      : "=r"(c.v.x), "=r"(c.v.y), "=r"(c.v.z), "=r"(c.v.w)
      : "l"(p), "r"((int)on));
  return c;
}

// Pass A's copies.  A warp of pass A samples patches of 8 (y) x 4 (x) voxels of one plane, and what a
// warp-wide cell load costs is one L1 wavefront per distinct 128-byte line.  Cells (X, Y, Z), each
// coordinate one more than the cell's lower corner, are stored as bricks of 2 (y) x 2 (z) cells, y
// fastest, then x: over random rotations such a patch touches 18.7 lines (FP32; 15.9 with BF16
// cells), a row of 32 voxels over cells in plain order 26.8.
__host__ __device__ constexpr unsigned brick_row(int n) { return 4u * (unsigned)((n + 2) / 2); }  // cells per X
__host__ __device__ constexpr unsigned brick_slab(int n) { return brick_row(n) * (unsigned)(n + 1); }  // per Z pair
__host__ __device__ constexpr long brick_cells(int n) { return (long)brick_slab(n) * ((n + 2) / 2); }
__host__ __device__ constexpr unsigned brick_index(int n, unsigned X, unsigned Y, unsigned Z) {
  return (Z >> 1) * brick_slab(n) + X * brick_row(n) + (Y >> 1) * 4u + (Z & 1u) * 2u + (Y & 1u);
}
// The mask in tiles of one patch: a warp reads one 128-byte line.
__host__ __device__ constexpr int mask_tile_index(int n, int x, int y, int z) {
  return ((z * (n / 4) + x / 4) * (n / 8) + y / 8) * 32 + (x % 4) * 8 + y % 8;
}

template <typename T>
__device__ __forceinline__ CellT<T> make_cell(const float* __restrict__ vol, int n, int i, int j, int k) {
  float v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int x = i + (q & 1), y = j + ((q >> 1) & 1), z = k + ((q >> 2) & 1);
    v[q] = (x >= 0 && y >= 0 && z >= 0 && x < n && y < n && z < n) ? vol[((long)z * n + y) * n + x] : 0.f;
  }
  CellT<T> c;
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<CellT<float>&>(c).lo = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<CellT<float>&>(c).hi = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&reinterpret_cast<CellT<__nv_bfloat16>&>(c).v);
#pragma unroll
    for (int q = 0; q < 4; ++q) p[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
  }
  return c;
}

// Builds the corner cells of an n^3 FP32 volume, stored as T, x fastest.
template <typename T>
__global__ void k_build_cells(const float* __restrict__ vol, int n, CellT<T>* __restrict__ cells) {
  const long nc = n + 1;
  const long total = nc * nc * nc;
  for (long ci = blockIdx.x * (long)blockDim.x + threadIdx.x; ci < total; ci += (long)gridDim.x * blockDim.x)
    cells[ci] = make_cell<T>(vol, n, (int)(ci % nc) - 1, (int)((ci / nc) % nc) - 1, (int)(ci / (nc * nc)) - 1);
}
// The same cells as bricks.
template <typename T>
__global__ void k_build_bricks(const float* __restrict__ vol, int n, CellT<T>* __restrict__ cells) {
  const long total = brick_cells(n);
  const long row = brick_row(n), slab = brick_slab(n);
  for (long ci = blockIdx.x * (long)blockDim.x + threadIdx.x; ci < total; ci += (long)gridDim.x * blockDim.x) {
    const int Z = 2 * (int)(ci / slab) + (int)((ci >> 1) & 1), X = (int)(ci % slab / row);
    const int Y = 2 * (int)(ci % row / 4) + (int)(ci & 1);
    cells[ci] = make_cell<T>(vol, n, X - 1, Y - 1, Z - 1);
  }
}
static __global__ void k_mask_tiles(const float* __restrict__ mask, int n, float* __restrict__ tiles) {
  const int total = n * n * n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
    tiles[mask_tile_index(n, i % n, (i / n) % n, i / (n * n))] = mask[i];
}

struct EvalItem {
  int particle;
  int orient;          // global orientation index
};

struct EvalStats {
  double sum_r, sum_r2, energy_spec, pad;
};

// Result of one evaluation: normalised CC at the peak and the integer shift.
struct EvalResult {
  float cc;
  int peak[3];
};

struct SearchChunkArgs {
  const EvalItem* items;     // [E]
  const DevParticle* parts;
  const DevRef* refs;
  const double* dmat;        // [norient][9] column-major defineMatrix([phi,theta,psi-phi],'inv')
  float2* s1;                // [E][ky][z][column], S1_EVAL per evaluation
  float2* s2;                // [E][w][lpos(ky)][PC] planes, S2_PLANE each
  EvalStats* stats;          // [E]
  unsigned long long* keys;  // [E]
  int n_items;
  int planes;                // z-planes per pass-A CTA
  int radius;
  int interp;
  // With `done` set, the last pass-C CTA of an evaluation decodes it into results / best_keys
  // and clears its stats, key and counter for the next chunk.
  unsigned* done = nullptr;                  // [E] pass-C CTAs finished
  EvalResult* results = nullptr;             // [total evaluations of the run]
  unsigned long long* best_keys = nullptr;   // [particles]
  // Bounded device-side waits: a wait that gives up after wait_cycles SM clock cycles ORs
  // kStatusWaitTimeout into *status (when set) and its CTA returns without a result.
  unsigned* status = nullptr;
  long long wait_cycles = 1ll << 31;         // about a second at the B200's 1.965 GHz
  unsigned phantom_tx = 0;                   // test hook: bytes announced but never copied (0)
};
constexpr unsigned kStatusWaitTimeout = 1u;

// Decodes evaluation e of a chunk from its peak key and folds it into its particle's
// best-orientation key (cc, then the first orientation on ties).
__device__ __forceinline__ void decode_eval(const SearchChunkArgs& a, int n, int e, unsigned long long key) {
  const EvalItem it = a.items[e];
  const DevParticle& pt = a.parts[it.particle];
  EvalResult r;
  const int c = n / 2;
  if (key == 0ull) {
    r.cc = __int_as_float(0x7fc00000);
    r.peak[0] = r.peak[1] = r.peak[2] = 0;
  } else {
    r.cc = key_to_float((unsigned int)(key >> 32));
    const unsigned int lin = 0xffffffffu - (unsigned int)(key & 0xffffffffull);
    r.peak[0] = (int)(lin % n) - c;
    r.peak[1] = (int)((lin / n) % n) - c;
    r.peak[2] = (int)(lin / ((unsigned)n * n)) - c;
  }
  a.results[pt.eval_base + (it.orient - pt.orient_begin)] = r;
  if (key != 0ull) {
    const unsigned long long bk = ((unsigned long long)ordered_key(r.cc) << 32) | (0xffffffffu - (unsigned)it.orient);
    atomicMax(a.best_keys + it.particle, bk);
  }
}

// z-planes per pass-A CTA: 1, 2, 4 or 8 at 64^3, up to 4 at 96^3, up to 2 at 128^3.
__host__ __device__ constexpr bool planes_allowed(int N, int g) {
  return (g == 1 || g == 2 || g == 4 || g == 8) && g <= (N <= 64 ? 8 : N <= 96 ? 4 : 2);
}

// How pass A samples: the two trilinear modes through the cells, the same from the plain volume (a caller
// without cells), or tricubic from the plain volume.
enum Gather { kGatherCells, kGatherPlain, kGatherCubic };

// The line transforms of passes A and B split N = 8 R2: with n = j + R2 r and k = k1 + 8 k2,
//   X(k) = DFT_R2 over j of [ w_N^(j k1) DFT_8 over r of x(j + R2 r) ],
// so a thread holds one 8-point or one R2-point butterfly of its own line, neighbouring threads hold
// neighbouring lines (shared memory is read and written in consecutive words, whatever the axis), all
// threads of a warp use the same twiddles, and between the two stages the data crosses shared memory
// once, in place: the R2-point stage reads and writes the slots (k1, 0 .. R2-1) that no other thread
// touches.  (Teams of 8 lanes transforming one line each crossed it three to four times per axis.)
template <int N>
struct SearchCfg {
  static constexpr int NH = N / 2 + 1;
  static constexpr int P = team_size(N);
  static constexpr int R2 = N / 8;
  // ---- pass A.  A plane's lines are its N/2 row pairs (y, y + N/2) along x, then its N/2 columns along
  // y (columns 0 and N/2, both real after x, share one).  Element (k1, m) of line q lives at
  // k1 XA + m XB + q: with XB = 8 and XA = 1 (mod 16 slots of 8 bytes) a half-warp falls on distinct
  // banks in the gather's patches (8 q x 2 m) and in the y stages, whose sixteen neighbouring columns
  // kx read slots (kx mod 8, kx / 8) or their mirrors.
  static constexpr int Q = N / 2;
  static constexpr int XB = Q + 8;
  static constexpr int XA = R2 * XB + 1;
  static_assert(XB % 16 == 8 && XA % 16 == 1 && Q % 8 == 0, "bank layout");
  static constexpr int NT_A = N == 96 ? 192 : 256;
  static constexpr int JA = NT_A / Q;            // butterflies of a line formed side by side
  static_assert(NT_A % Q == 0 && R2 % JA == 0 && 8 % JA == 0 && JA % 4 == 0, "whole rounds and patches");
  static constexpr size_t SMEM_A = sizeof(float2) * (8 * (size_t)XA + N + N);
  // Resident pass-A CTAs asked of the compiler, and cells in flight per thread (2 UNROLL_A): at 64^3 two
  // and four CTAs per SM (1,095 ns per evaluation; four and three CTAs 1,150), at 96^3 and 128^3 four
  // (3,490 and 9,180 ns; two: 3,760 and 10,760).  Four at one CTA more spill and lose by a third: local
  // memory shares the L1 that the gather streams through.  The tricubic sampler's 64 loads want more
  // registers at 64^3 (64 masked orientations: 683 us at three CTAs, 715 at four, 731 at two).
  static constexpr int UNROLL_A = N == 64 ? 1 : 2;
  static constexpr int min_blocks_a(Gather g) { return N > 96 ? 2 : N == 64 && g == kGatherCubic ? 3 : 4; }
  // ---- pass B: the z lines of one ky, the R2-point stage first (its inputs come straight from global
  // memory) and the 8-point one second, so that the product needs 8 spectrum and weight elements per
  // butterfly.  S1 rows hold column N/2 first, then 0 .. N/2-1, padded to whole 32-byte sectors;
  // element (k1, j) of column c lives at k1 ZA + j TP + c, and thread t has column t % TP, so that both
  // stages' accesses are consecutive in t.
  static constexpr int TP = (NH + 3) / 4 * 4;
  static constexpr int JB = N == 64 ? 8 : 4;
  static constexpr int NT_B = (TP * JB + 31) / 32 * 32;
  static constexpr int ZA = 8 * TP + (16 - (7 * TP) % 16) % 16;
  static_assert((ZA - TP) % 16 == 0 && R2 % JB == 0 && 8 % JB == 0, "bank layout, whole rounds");
  static constexpr int EVALS_B = N <= 96 ? 4 : 2;
  static constexpr int MINB_B = N == 128 ? 2 : 3;
  static constexpr size_t SMEM_B = sizeof(float2) * (R2 * (size_t)ZA + N);
  static constexpr size_t S1_EVAL = (size_t)N * N * TP;
  // ---- pass C uses half as many teams as the y transforms have lines (two rounds of y lines), so
  // that the C2R phase, where (2 r + 1 + 1) / 2 row pairs (8 at r = 7) keep as many teams busy,
  // leaves fewer idle and more CTAs fit per SM: 64^3 20 teams of 8 lanes, six CTAs per SM at 64
  // registers (88.7 us per 602-evaluation chunk against 131.1 with 33 teams); 96^3 28 teams and
  // 128^3 36, where the whole-row CTAs (416 and 544 threads) fitted once per SM by registers
  static constexpr int NT_BC = ((NH * P / 2 + 31) / 32) * 32;
  static constexpr int MINB_C = N <= 64 ? 6 : 2;
  static constexpr int TEAMS_BC = NT_BC / P;
  // FFT lines use padded positions (lpos<1>): a strided line of N elements spans PY rows, a
  // contiguous line buffer LP slots; LP = 8 (mod 16) puts neighbouring teams 16 banks apart.
  static constexpr int PY = padded_len(N);
  static constexpr int LP = PY + ((8 - PY % 16) + 16) % 16;
  static constexpr int TEAMS_LC = 16;  // (2 r + 1 + 1) / 2 <= 16 row pairs for r <= 15
  static_assert(TEAMS_BC >= TEAMS_LC, "pass C needs a team for every line buffer");
  // Pass C's tile: S2 planes are written by pass B in this layout (rows ky at lpos<1>(ky), even
  // pitch PC), so pass C brings a plane in with one bulk copy; its y transforms then take
  // consecutive columns (a bank model gives the same wavefronts as the odd pitch with paired
  // columns).
  static constexpr int PC = NH + (NH & 1);
  static constexpr size_t S2_PLANE = (size_t)PY * PC;
  static constexpr size_t SMEM_C = sizeof(float2) * (S2_PLANE + N + (size_t)TEAMS_LC * LP);
};

// S1 elements per evaluation of box n.
inline size_t s1_eval_elems(int n) {
  return n == 64 ? SearchCfg<64>::S1_EVAL : n == 96 ? SearchCfg<96>::S1_EVAL : SearchCfg<128>::S1_EVAL;
}
// S2 elements per output plane of box n (pass C's tile layout).
inline size_t s2_plane_elems(int n) {
  return n == 64 ? SearchCfg<64>::S2_PLANE : n == 96 ? SearchCfg<96>::S2_PLANE : SearchCfg<128>::S2_PLANE;
}

template <typename Tv>
__device__ __forceinline__ Tv block_sum(Tv v, Tv* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  Tv t = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  return t;  // valid in thread 0
}

// max of |a|, |b|, |c|; NaN when any is NaN.
__device__ __forceinline__ float max_abs_nan(float a, float b, float c) {
  float d;
  asm("{\n .reg .f32 x, y, z;\n abs.f32 x, %1;\n abs.f32 y, %2;\n abs.f32 z, %3;\n max.NaN.f32 x, x, y;\n"
      " max.NaN.f32 %0, x, z;\n}\n"
      : "=f"(d)
      : "f"(a), "f"(b), "f"(c));
  return d;
}

// Same interpolation order as sample_linear, so both paths give identical results.
__device__ __forceinline__ float cell_trilinear(const float v[8], const float f[3]) {
  const float c00 = fmaf(f[0], v[1] - v[0], v[0]), c10 = fmaf(f[0], v[3] - v[2], v[2]);
  const float c01 = fmaf(f[0], v[5] - v[4], v[4]), c11 = fmaf(f[0], v[7] - v[6], v[6]);
  const float c0 = fmaf(f[1], c10 - c00, c00), c1 = fmaf(f[1], c11 - c01, c01);
  return fmaf(f[2], c1 - c0, c0);
}

// The reference's value at the sampling point of voxel (u, v, w) (from the centre) under the matrix rows m,
// for the modes without cells.
template <Gather GATHER, typename T>
__device__ __forceinline__ float sample_plain(int mode, const T* __restrict__ src, int n, const float* __restrict__ m,
                                              float u, float v, float w) {
  const float c = (float)(n / 2);
  const float sx = fmaf(m[0], u, fmaf(m[1], v, m[2] * w)) + c, sy = fmaf(m[3], u, fmaf(m[4], v, m[5] * w)) + c,
              sz = fmaf(m[6], u, fmaf(m[7], v, m[8] * w)) + c;
  return GATHER == kGatherCubic ? sample_cubic(src, n, n, n, sx, sy, sz)
         : mode == EMC_INTERP_LINEAR_BORDER ? sample_linear_border(src, n, n, n, sx, sy, sz)
                                            : sample_linear(src, n, n, n, sx, sy, sz);
}

// ------------------------------------------------------------------ pass A
// One z-plane after another: thread (q, j) samples the voxels x = j + R2 r (r = 0..7) of rows q and
// q + N/2, whose pairs are the inputs of its first x butterfly, so the rotated plane crosses shared
// memory only in the thread's own slots.  A warp takes 8 rows x 4 columns of the plane and reads the
// cells from bricks (see brick_index); floors by a round-down addition (kFloorMagic).
//
// GATHER: see Gather.
template <int N, typename T, Gather GATHER>
__global__ void __launch_bounds__(SearchCfg<N>::NT_A, SearchCfg<N>::min_blocks_a(GATHER)) k_search_fwd_xy(
    const SearchChunkArgs a, const float2* __restrict__ g_tw) {
  using C = SearchCfg<N>;
  constexpr int R2 = C::R2, Q = C::Q, XA = C::XA, XB = C::XB, JA = C::JA;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* buf = reinterpret_cast<float2*>(smem_raw);  // [8][XA]
  float2* s_tw = buf + 8 * XA;                         // [N]
  float2* s_col = s_tw + N;                            // [N], the packed columns 0 and N/2 after y
  __shared__ float s_m[9];
  __shared__ double red[2][32];

  const int e = blockIdx.y;
  if (e >= a.n_items) return;
  const EvalItem it = a.items[e];
  const DevParticle& pt = a.parts[it.particle];
  const DevRef rf = a.refs[pt.ref];
  load_twiddles<N>(s_tw, g_tw);
  if (threadIdx.x < 9) {
    // sampling matrix rows of RotMat' with RotMat = prior * D (FP64 composition): entry (i, j) is
    // RotMat(j, i) = sum_k prior(j, k) D(k, i)
    const int i = threadIdx.x / 3, j = threadIdx.x % 3;
    const double* d = a.dmat + 9L * it.orient;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) acc = fma(pt.prior[j + 3 * k], d[k + 3 * i], acc);
    s_m[threadIdx.x] = (float)acc;
  }
  __syncthreads();
  const bool weighted = rf.wref || pt.wedge;
  const CellT<T>* __restrict__ cells = reinterpret_cast<const CellT<T>*>(rf.bricks);
  // samples with |s - (N-1)/2| <= lim on every axis are inside (0 <= s <= N-1, or -1 < s < N)
  constexpr float h = 0.5f * (N - 1);
  const float lim = a.interp == EMC_INTERP_LINEAR_BORDER ? __int_as_float(__float_as_int(h + 1.f) - 1) : h;
  const int q = threadIdx.x % Q, jt = threadIdx.x / Q;
  constexpr int c = N / 2;
  // shared-memory column of the y stages: kx = q, its mirror N - kx (N/2 for the packed column 0)
  const int mir = q == 0 ? Q : N - q;
  const int slot_k = (q & 7) * XA + (q >> 3) * XB, slot_m = (mir & 7) * XA + (mir >> 3) * XB;
  double sum1 = 0.0, sum2 = 0.0;
  // First x stage of a butterfly whose inputs lie in this thread's slots, in place.  Without a weight on the
  // reference its real-space sums are formed here, in FP64 from the samples on: E_R cancels for a
  // reference with an offset (FP32 sums over a thread's samples put the CC at a mean of 100 sigma off by
  // up to 6e-5, depending on the plane count; now 1e-7 at every count).  Here and not in the gather,
  // whose registers are all taken; weighted searches skip it, unweighted ones take at most 3 % longer.
  auto first_x_stage = [&](float2* own) {
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = own[r * XA];
    if (!weighted) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const double va = v[r].x, vb = v[r].y;
        sum1 += va + vb;
        sum2 = fma(va, va, fma(vb, vb, sum2));
      }
    }
    Dft<8, -1>::run(v);
#pragma unroll
    for (int r = 0; r < 8; ++r) own[r * XA] = v[r];
  };

#pragma unroll 1
  for (int z = blockIdx.x * a.planes; z < (int)(blockIdx.x + 1) * a.planes; ++z) {
    // 1. gather and the first x stage, rows gq and gq + N/2
    {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      const int gq = (lane & 7) + 8 * (warp % (Q / 8)), gj = (lane >> 3) + 4 * (warp / (Q / 8));
      const float tx = pt.shift[0], pw = (float)(z - c) - pt.shift[2];
      const float pva = (float)(gq - c) - pt.shift[1], pvb = (float)(gq + Q - c) - pt.shift[1];
      if constexpr (GATHER == kGatherCells) {
        constexpr int U = C::UNROLL_A;
        float base[2][3], mx[3];  // sample points at u = 0 of the two rows
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float w = s_m[3 * i + 2] * pw;
          base[0][i] = fmaf(s_m[3 * i + 1], pva, w) + (float)c;
          base[1][i] = fmaf(s_m[3 * i + 1], pvb, w) + (float)c;
          mx[i] = s_m[3 * i];
        }
        // the rows' x extents of non-zero mask voxels: the samples outside need no cell
        int lo[2], len[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const unsigned ext = rf.mask_rows ? __ldg(rf.mask_rows + z * N + gq + k * Q) : (unsigned)N << 16;
          lo[k] = (int)(ext & 0xffffu);
          len[k] = (int)(ext >> 16) - lo[k];
        }
        const float* mask = rf.mask_tiles ? rf.mask_tiles + mask_tile_index(N, lane >> 3, gq, z) : nullptr;
#pragma unroll 1
        for (int j = gj; j < R2; j += JA) {
          // U r (2 U cells in flight) per step, the samples left in the thread's own slots: a rolled
          // loop, since the compiler otherwise starts all sixteen loads at once and spills
          float2* own = buf + j * XB + gq;
          float xj = (float)(j - c);
          int x = j;
#pragma unroll 1
          for (int r0 = 0; r0 < 8; r0 += U, x += U * R2, xj += (float)(U * R2), own += U * XA) {
            CellT<T> cell[U][2];
            float f[U][2][3], mk[U][2];
            bool ok[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const float pu = (xj + (float)(R2 * u)) - tx;
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                float off[3];
                unsigned cc[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                  const float s = fmaf(mx[i], pu, base[k][i]);
                  const float fl = __fadd_rd(s, kFloorMagic);
                  f[u][k][i] = s - (fl - kFloorMagic);
                  off[i] = s - h;
                  cc[i] = __float_as_uint(fl) + (1u - kFloorBits);
                }
                ok[u][k] = max_abs_nan(off[0], off[1], off[2]) <= lim && (unsigned)(x + R2 * u - lo[k]) < (unsigned)len[k];
                // brick_index(N, X, Y, Z)
                constexpr unsigned row = brick_row(N), half = brick_slab(N) / 2;
                const unsigned idx = cc[2] * half - (cc[2] & 1u) * (half - 2u) + cc[0] * row + 2u * cc[1] - (cc[1] & 1u);
                cell[u][k] = load_cell_if(cells + idx, ok[u][k]);
                // x / 4 advances the tile row, y / 8 the tile
                mk[u][k] = mask ? __ldg(mask + ((x + R2 * u) / 4 * (N / 8) + k * (Q / 8)) * 32) : 1.f;
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              float val[2];
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                float cv[8];
                cell_values(cell[u][k], cv);
                val[k] = ok[u][k] ? cell_trilinear(cv, f[u][k]) * mk[u][k] : 0.f;
              }
              own[u * XA] = make_float2(val[0], val[1]);
            }
          }
          first_x_stage(buf + j * XB + gq);
        }
      } else {
        // 32 consecutive voxels of a row per warp: the plain volume is x fastest, so their loads share lines
        // where the patches' rows do not.  (64 tricubic orientations near the identity: 64^3 1,039 -> 683 us,
        // 96^3 3,588 -> 2,824, 128^3 9,196 -> 5,945 against one call of the sampler per voxel of a patch.)
        const T* src = reinterpret_cast<const T*>(rf.data);
        const float* mask = rf.mask ? rf.mask + (long)z * N * N : nullptr;
        for (int i = threadIdx.x; i < N * N; i += C::NT_A) {
          const int x = i % N, y = i / N;
          float v = sample_plain<GATHER>(a.interp, src, N, s_m, (float)(x - c) - tx, (float)(y - c) - pt.shift[1], pw);
          if (mask) v *= __ldg(mask + i);
          reinterpret_cast<float*>(buf + (x / R2) * XA + (x % R2) * XB + y % Q)[y / Q] = v;
        }
        __syncthreads();
#pragma unroll 1
        for (int j = gj; j < R2; j += JA) first_x_stage(buf + j * XB + gq);
      }
    }
    __syncthreads();
    // 2. second x stage: Z(k1 + 8 k2) of every row pair, left at (k1, k2)
#pragma unroll 1
    for (int k1 = jt; k1 < 8; k1 += JA) {
      float2* line = buf + k1 * XA + q;
      float2 v[R2];
#pragma unroll
      for (int m = 0; m < R2; ++m) v[m] = line[m * XB];
#pragma unroll
      for (int m = 1; m < R2; ++m) v[m] = cmul(v[m], s_tw[m * k1]);
      Dft<R2, -1>::run(v);
#pragma unroll
      for (int m = 0; m < R2; ++m) line[m * XB] = v[m];
    }
    __syncthreads();
    // 3. first y stage of column kx = q: rows y = j + R2 r from the Hermitian split of the row pairs
    // y, y + N/2 = (r, r + 4).  Columns 0 and N/2 of a row are real and share a column as (X(0), X(N/2)).
    // The pairs' entries kx and N - kx are this column's alone: the results go back into them.
#pragma unroll 1
    for (int j = jt; j < R2; j += JA) {
      float2* pk = buf + slot_k + j;
      float2* pm = buf + slot_m + j;
      float2 v[8];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 zk = pk[R2 * r], zm = pm[R2 * r];
        if (q == 0) {
          v[r] = make_float2(zk.x, zm.x);
          v[r + 4] = make_float2(zk.y, zm.y);
        } else {
          v[r] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
          v[r + 4] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
        }
      }
      Dft<8, -1>::run(v);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        pk[R2 * r] = v[r];
        pm[R2 * r] = v[r + 4];
      }
    }
    __syncthreads();
    // 4. second y stage, straight to S1 (columns 1 .. N/2-1); the packed column to shared memory
    float2* s1 = a.s1 + (size_t)e * C::S1_EVAL + (size_t)z * C::TP;
#pragma unroll 1
    for (int k1 = jt; k1 < 8; k1 += JA) {
      const float2* col = buf + (k1 < 4 ? slot_k : slot_m) + R2 * (k1 & 3);
      float2 v[R2];
#pragma unroll
      for (int m = 0; m < R2; ++m) v[m] = col[m];
#pragma unroll
      for (int m = 1; m < R2; ++m) v[m] = cmul(v[m], s_tw[m * k1]);
      Dft<R2, -1>::run(v);
      if (q == 0) {
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) s_col[k1 + 8 * k2] = v[k2];
      } else {
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) s1[(size_t)(k1 + 8 * k2) * N * C::TP + 1 + q] = v[k2];
      }
    }
    __syncthreads();
    // columns N/2 and 0 from the packed one: with Z = F(X(0) + i X(N/2)),
    // F X(0)(y) = (Z(y) + conj Z(-y)) / 2 and F X(N/2)(y) = (Z(y) - conj Z(-y)) / 2i
    if (threadIdx.x < N) {
      const float2 zp = s_col[threadIdx.x], zm = s_col[(N - threadIdx.x) % N];
      *reinterpret_cast<float4*>(s1 + (size_t)threadIdx.x * N * C::TP) =
          make_float4(0.5f * (zp.y + zm.y), -0.5f * (zp.x - zm.x), 0.5f * (zp.x + zm.x), 0.5f * (zp.y - zm.y));
    }
  }
  if (!weighted) {
    // E_R from the real-space sums (Parseval) is needed only without a weight on the reference; with
    // one, pass B forms the weighted spectral energy (the branch is uniform over the block)
    double t1 = block_sum(sum1, red[0]);
    double t2 = block_sum(sum2, red[1]);
    if (threadIdx.x == 0) {
      atomicAdd(&a.stats[e].sum_r, t1);
      atomicAdd(&a.stats[e].sum_r2, t2);
    }
  }
}

// ------------------------------------------------------------------ pass B
// Outputs 0 and R - 1 of an inverse R-point transform; tw8: w_N^(8 k) = e^(-2 pi i k / R) at index 8 k.
template <int R>
__device__ __forceinline__ void idft_ends(const float2 v[R], const float2* tw8, float2& first, float2& last) {
  float2 s[R / 2], d[R / 2];
#pragma unroll
  for (int k = 0; k < R / 2; ++k) {
    s[k] = cadd(v[k], v[k + R / 2]);
    d[k] = csub(v[k], v[k + R / 2]);  // e^(-2 pi i k / R) changes sign from k to k + R / 2
  }
  if constexpr (R == 8) {
    first = cadd(cadd(s[0], s[2]), cadd(s[1], s[3]));
    const float2 p = csub(d[1], d[3]), t = cadd(d[1], d[3]);  // e^(-i pi/4) d1 + e^(-3 i pi/4) d3
    last.x = d[0].x + d[2].y + EMC_SQRT1_2 * (p.x + t.y);
    last.y = d[0].y - d[2].x + EMC_SQRT1_2 * (p.y - t.x);
  } else {
    float2 s0 = cadd(s[0], s[1]), s1 = cadd(s[2], s[3]), e0 = d[0], e1 = cmul(d[1], tw8[8]);
#pragma unroll
    for (int k = 4; k < R / 2; k += 2) {
      s0 = cadd(s0, s[k]);
      s1 = cadd(s1, s[k + 1]);
    }
#pragma unroll
    for (int k = 2; k < R / 2; k += 2) {
      e0 = cadd(e0, cmul(d[k], tw8[8 * k]));
      e1 = cadd(e1, cmul(d[k + 1], tw8[8 * (k + 1)]));
    }
    first = cadd(s0, s1);
    last = cadd(e0, e1);
  }
}

// The z lines of one ky for EVALS_B consecutive evaluations (consecutive orientations of one
// particle, but at a particle boundary).  A butterfly's spectrum and weight elements are asked for a
// stage before its product needs them; at 64^3, where a thread has one butterfly, they stay in
// registers while the particle does not change.
template <int N>
__global__ void __launch_bounds__(SearchCfg<N>::NT_B, SearchCfg<N>::MINB_B) k_search_z_mul(
    const SearchChunkArgs a, const float2* __restrict__ g_tw) {
  using C = SearchCfg<N>;
  constexpr int R2 = C::R2, TP = C::TP, ZA = C::ZA, JB = C::JB, NH = C::NH;
  constexpr bool ONE = JB == R2;  // one butterfly of the second stage per thread
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* buf = reinterpret_cast<float2*>(smem_raw);  // [R2][ZA]
  float2* s_tw = buf + R2 * ZA;                        // [N]
  __shared__ double red[32];
  const int e_first = blockIdx.y * C::EVALS_B;
  if (e_first >= a.n_items) return;
  const int ne = min(C::EVALS_B, a.n_items - e_first);
  const int ky = blockIdx.x, w = 2 * a.radius + 1;
  const int col = threadIdx.x % TP, jt = threadIdx.x / TP;
  const int kx = col == 0 ? N / 2 : col - 1;
  const bool in = threadIdx.x < TP * JB, line = in && col < NH;  // whole warps' remainder, pad columns
  const double hw = (kx == 0 || 2 * kx == N) ? 1.0 : 2.0;
  constexpr size_t ZS = (size_t)N * NH;  // elements per z step of the spectrum and weight
  const size_t at = (size_t)ky * NH + (line ? kx : 0);
  // r < 8: of the last stage's R2 outputs only the first (z = m) and the last (z = m - 8) can lie in
  // the window
  const bool narrow = a.radius < 8;
  load_twiddles<N>(s_tw, g_tw);
  int loaded = -1;  // particle whose spectrum and weight are in the registers (ONE)
  float2 qr[8];
  float wr[8];
#pragma unroll 1
  for (int k = 0; k < ne; ++k) {
    const int e = e_first + k;
    const EvalItem it = a.items[e];
    const DevParticle& pt = a.parts[it.particle];
    // weights on the rotated reference (BH_multi_xcf_Translational_2.m:35-38): the particle's
    // wdgMask and the reference's bandpass wref
    const float* __restrict__ wref = a.refs[pt.ref].wref;
    const float* __restrict__ w1 = pt.wedge ? pt.wedge : wref;
    const float* __restrict__ w2 = pt.wedge ? wref : nullptr;
    const float2* __restrict__ spec = pt.spec;
    const bool weighted = w1 != nullptr;
    // spectrum and weight of butterfly k1 (kz = k1 + R2 k2)
    auto fetch = [&](int k1) {
#pragma unroll
      for (int k2 = 0; k2 < 8; ++k2) {
        const size_t i = (size_t)(k1 + R2 * k2) * ZS + at;
        qr[k2] = __ldg(spec + i);
        wr[k2] = w1 ? __ldg(w1 + i) : 1.f;
        if (w2) wr[k2] *= __ldg(w2 + i);
      }
    };
    __syncthreads();  // the previous evaluation is done with the buffer (and the twiddles are there)
    const float2* s1 = a.s1 + (size_t)e * C::S1_EVAL + (size_t)ky * N * TP + col;
    // first stage, from global memory: z = j + 8 r
    if (in) {
#pragma unroll 1
      for (int j = jt; j < 8; j += JB) {
        float2 v[R2];
#pragma unroll
        for (int r = 0; r < R2; ++r) v[r] = __ldcs(s1 + (size_t)(j + 8 * r) * TP);
        Dft<R2, -1>::run(v);
#pragma unroll
        for (int k1 = 0; k1 < R2; ++k1) buf[k1 * ZA + j * TP + col] = v[k1];
      }
    }
    if (line && (!ONE || it.particle != loaded)) fetch(jt);
    loaded = it.particle;
    __syncthreads();
    // second stage, product, first inverse stage: kz = k1 + R2 k2 in registers
    double ed = 0.0;  // |.|^2 of this thread's elements: a butterfly's eight in FP32, then FP64
    if (line) {
#pragma unroll 1
      for (int k1 = jt; k1 < R2; k1 += JB) {
        float2* lp = buf + k1 * ZA + col;
        float2 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = lp[j * TP];
#pragma unroll
        for (int j = 1; j < 8; ++j) v[j] = cmul(v[j], s_tw[j * k1]);
        Dft<8, -1>::run(v);
        float ef = 0.f;
#pragma unroll
        for (int k2 = 0; k2 < 8; ++k2) {
          const bool origin = k1 + R2 * k2 + ky + kx == 0;
          float2 r = v[k2];
          if (weighted) {
            r.x *= wr[k2];
            r.y *= wr[k2];
            if (!origin) ef = fmaf(r.x, r.x, fmaf(r.y, r.y, ef));
          }
          const float2 x = cmulc(qr[k2], r);
          v[k2] = origin ? make_float2(0.f, 0.f) : x;
        }
        ed += (double)ef;
        if (!ONE && k1 + JB < R2) fetch(k1 + JB);
        Dft<8, 1>::run(v);
#pragma unroll
        for (int m = 1; m < 8; ++m) v[m] = cmulc(v[m], s_tw[m * k1]);
#pragma unroll
        for (int m = 0; m < 8; ++m) lp[m * TP] = v[m];
      }
    }
    if (weighted) {
      const double t = block_sum(line ? hw * ed : 0.0, red);  // (synchronises)
      if (threadIdx.x == 0) atomicAdd(&a.stats[e].energy_spec, t);
    } else {
      __syncthreads();
    }
    // last inverse stage: z = m + 8 l, the planes |sz| <= r to S2
    if (line) {
      float2* dst = a.s2 + (size_t)e * w * C::S2_PLANE + (size_t)lpos<1>(ky) * C::PC + kx;
#pragma unroll 1
      for (int m = jt; m < 8; m += JB) {
        float2 v[R2];
#pragma unroll
        for (int k1 = 0; k1 < R2; ++k1) v[k1] = buf[k1 * ZA + m * TP + col];
        if (narrow) {
          float2 first, last;
          idft_ends<R2>(v, s_tw, first, last);
          if (m <= a.radius) dst[(size_t)(m + a.radius) * C::S2_PLANE] = first;
          if (8 - m <= a.radius) dst[(size_t)(m - 8 + a.radius) * C::S2_PLANE] = last;
        } else {
          Dft<R2, 1>::run(v);
#pragma unroll
          for (int l = 0; l < R2; ++l) {
            const int z = m + 8 * l, sz = z < N / 2 ? z : z - N;
            if (abs(sz) <= a.radius) dst[(size_t)(sz + a.radius) * C::S2_PLANE] = v[l];
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------ pass C
template <int N>
__global__ void __launch_bounds__(SearchCfg<N>::NT_BC, SearchCfg<N>::MINB_C) k_search_inv_peak(const SearchChunkArgs a,
                                                                          const float2* __restrict__ g_tw) {
  using C = SearchCfg<N>;
  constexpr int NH = C::NH, P = C::P;
  constexpr int PC = C::PC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tile = reinterpret_cast<float2*>(smem_raw);   // [PY][PC], row y at lpos<1>(y)
  float2* s_tw = tile + C::S2_PLANE;
  float2* lines = s_tw + N;                              // [TEAMS][LP]
  __shared__ unsigned long long s_best;
  __shared__ uint64_t bar;
  constexpr unsigned PLANE_BYTES = (unsigned)(sizeof(float2) * C::S2_PLANE);
  static_assert(PLANE_BYTES % 16 == 0, "bulk copy size");

  const int e = blockIdx.y;
  if (e >= a.n_items) return;
  const int j = blockIdx.x;
  const int r = a.radius, w = 2 * r + 1;
  const int sz = j - r;
  const EvalItem it = a.items[e];
  const DevParticle& pt = a.parts[it.particle];
  // with a weight on the reference E_R is its weighted spectral energy (pass B), else the
  // DC-free real-space energy of the rotated, masked reference (pass A, by Parseval)
  const bool weighted = a.refs[pt.ref].wref != nullptr || pt.wedge != nullptr;

  // the plane (pass B wrote it in this tile's layout) with one bulk copy, on a bounded wait
  if (threadIdx.x == 0) {
    s_best = 0ull;
    mbar_init(&bar, 1);
    mbar_arrive_expect_tx(&bar, PLANE_BYTES + a.phantom_tx);
    bulk_copy_g2s(tile, a.s2 + ((size_t)e * w + j) * C::S2_PLANE, PLANE_BYTES, &bar);
  }
  load_twiddles<N>(s_tw, g_tw);
  __syncthreads();  // the barrier is initialised before anyone polls it
  const bool arrived = mbar_wait(&bar, 0, a.wait_cycles);
  if (__syncthreads_or(!arrived)) {
    // the copy did not complete in time: report, give it a second bounded wait, and leave
    if (threadIdx.x == 0 && a.status) atomicOr(a.status, kStatusWaitTimeout);
    mbar_wait(&bar, 0, a.wait_cycles);
    return;
  }
  const int team = threadIdx.x / P, lane = threadIdx.x % P;
  LineTw<N, P> tc;
  tc.init(s_tw, lane);
  for (int base = 0; base < NH; base += C::TEAMS_BC) {
    const int li = base + team;  // consecutive columns for the teams of a warp
    fft_line<N, 1, P, 1>(tile + (li < NH ? li : 0), PC, lane, s_tw, li < NH, &tc);
  }
  __syncthreads();

  const EvalStats st = a.stats[e];
  const double er = weighted ? st.energy_spec : ((double)N * N * N * st.sum_r2 - st.sum_r * st.sum_r);
  const double denom = er * pt.energy;
  const float inv_norm = denom > 0.0 ? (float)(1.0 / sqrt(denom)) : 0.f;
  constexpr int c = N / 2;

  unsigned long long best = 0ull;
  // (warps with no row pair run the C2R loop predicated off; letting them skip it measured slower:
  // 74.2 -> 76-78 us per 64^3 chunk, a 4-byte spill and the branch against idle issue slots)
  const int npairs = (w + 1) / 2;
  const bool has_line = team < C::TEAMS_LC;
  float2* buf = lines + (size_t)(has_line ? team : 0) * C::LP;
  for (int base = 0; base < npairs; base += C::TEAMS_LC) {
    const int pr = base + team;
    const bool active = has_line && pr < npairs;
    const int ja = 2 * pr, jb = 2 * pr + 1;
    const bool has_b = jb < w;
    const int ya = (ja - r + N) % N, yb = has_b ? (jb - r + N) % N : ya;
    const float2* ra = tile + (size_t)lpos<1>(ya) * PC;
    const float2* rb = tile + (size_t)lpos<1>(yb) * PC;
    // Hermitian extension of rows a and b packed as a + i b
    fft_line_in<N, 1, P, 1>(
        [&](int n) {
          const bool lower = n <= N / 2;
          const int k = lower ? n : N - n;
          float2 A = ra[k];
          float2 B = has_b ? rb[k] : make_float2(0.f, 0.f);
          if (k == 0 || 2 * k == N) { A.y = 0.f; B.y = 0.f; }
          if (!lower) { A.y = -A.y; B.y = -B.y; }
          return make_float2(A.x - B.y, A.y + B.x);
        },
        buf, 1, lane, s_tw, active, &tc);
    if (active) {
      for (int t = lane; t < 2 * w; t += P) {
        const int which = t / w;  // 0: row a, 1: row b
        if (which == 1 && !has_b) continue;
        const int sx = (t % w) - r;
        const int sy = (which ? jb : ja) - r;
        if (sx * sx + sy * sy + sz * sz > r * r) continue;
        const float2 zv = buf[lpos<1>((sx + N) % N)];
        const float v = (which ? zv.y : zv.x) * inv_norm;
        if (v != v) continue;  // NaN never wins (MATLAB max ignores NaN)
        const unsigned int lin = (unsigned int)(((sz + c) * N + (sy + c)) * N + (sx + c));
        const unsigned long long key = ((unsigned long long)ordered_key(v) << 32) | (0xffffffffu - lin);
        best = key > best ? key : best;
      }
    }
    __syncwarp();
  }
  // block max
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax(&s_best, best);
  __syncthreads();
  if (threadIdx.x == 0 && s_best) atomicMax(&a.keys[e], s_best);
  if (a.done && threadIdx.x == 0) {
    // the last CTA of this evaluation (every other one has published its maximum) decodes it
    __threadfence();
    if (atomicAdd(&a.done[e], 1u) == (unsigned)(w - 1)) {
      __threadfence();
      const unsigned long long key = atomicExch(&a.keys[e], 0ull);
      decode_eval(a, N, e, key);
      a.stats[e] = EvalStats{0.0, 0.0, 0.0, 0.0};
      a.done[e] = 0u;
    }
  }
}

}  // namespace emc
