// FP32 CUDA-core kernels: expand, the likelihood / scaling / slice-average
// contractions as register-tiled FP32 kernels, softmax, insertion and model
// normalisation.  This is the plain-FP32 path of the engine and the engine
// behind the reference-compatible API in legacy.cu.
#include <cfloat>
#include <cstdint>

#include "fixed.cuh"
#include "insert.cuh"
#include "kernels.cuh"
#include "tile.cuh"
#include "voxel.h"

namespace emc {
namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of one double per thread over the block (blockDim.x multiple of 32).
__device__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < nw; ++i) s += red[i];
  return s;  // valid on thread 0
}

__device__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float s = -FLT_MAX;
  if (threadIdx.x == 0)
    for (int i = 0; i < nw; ++i) s = fmaxf(s, red[i]);
  return s;
}

// ------------------------------------------------------------------ expand --
// emc_cuda.cu:51-111 for the nearest mode (exclusive lower bound), trilinear
// otherwise.

// The nearest voxel (emc_voxel::nearest with lower bound 1) less one in each
// coordinate, false outside [1, side).  Rounding half away from zero is
// truncation of u + 1/2 where a voxel below 1 is outside anyway; that sum is
// rounded toward zero, so no u below a half reaches 1, and adding 2^23 leaves the
// whole number in the low bits.  Whatever is out of range, NaN included, gives a
// larger unsigned number.  Three instructions a coordinate, where roundf and its
// conversion to an integer (a unit that takes a warp every eight clocks) took
// seven: the expansion was bound by its instructions, 80 a pixel.  The same in
// the insertions and in the trilinear expansion changed nothing.
__device__ __forceinline__ bool nearest_from_1(const float* u, int side, uint32_t* k) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
    k[i] = __float_as_uint(__fadd_rz(__fadd_rz(u[i], 0.5f), 8388608.0f)) - 0x4b000001u;
  return max(max(k[0], k[1]), k[2]) < (uint32_t)(side - 1);
}

// Slice value W at continuous voxel position u (0 outside the grid).
template <int INTERP>
__device__ __forceinline__ float gather(const float* __restrict__ model, const float* u, int side) {
  if (INTERP == 0) {
    // rows of voxels fit 32 bits; the drop-in API has no bound on side^3
    uint32_t k[3];
    if (!nearest_from_1(u, side, k)) return 0.0f;
    const uint32_t row = (k[2] + 1) * (uint32_t)side + k[1] + 1;
    return __ldg(model + ((uint64_t)row * (uint32_t)side + k[0] + 1));
  }
  float acc = 0.0f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    int64_t v;
    float w;
    if (emc_voxel::trilinear_corner(u, side, c, &v, &w) && w != 0.0f)
      acc = fmaf(w, __ldg(model + v), acc);
  }
  return acc;
}

// Trilinear through the stencil table (launch_tri_table): the 8 corner values
// of base voxel floor(u) in one aligned 32-byte load, 0 for corners outside
// the grid.  The same FMAs in the same corner order as gather<1>: a corner
// that gather<1> skips (outside, or weight 0) adds w * 0 or 0 * value here,
// which leaves the sum unchanged, so the result is bit for bit the same.
__device__ __forceinline__ float gather_tri(const float4* __restrict__ tri, const float* u,
                                            int side) {
  const float fx = floorf(u[0]), fy = floorf(u[1]), fz = floorf(u[2]);
  const int x0 = (int)fx, y0 = (int)fy, z0 = (int)fz;
  if (x0 < -1 || x0 >= side || y0 < -1 || y0 >= side || z0 < -1 || z0 >= side) return 0.0f;
  const int64_t s1 = side + 1;
  const int64_t e = ((int64_t)(z0 + 1) * s1 + (y0 + 1)) * s1 + (x0 + 1);
  const float4 lo = __ldg(tri + 2 * e), hi = __ldg(tri + 2 * e + 1);
  const float val[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  const float ax = u[0] - fx, ay = u[1] - fy, az = u[2] - fz;
  float acc = 0.0f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int bx = c & 1, by = (c >> 1) & 1, bz = (c >> 2) & 1;
    const float w = (bx ? ax : 1.0f - ax) * (by ? ay : 1.0f - ay) * (bz ? az : 1.0f - az);
    acc = fmaf(w, val[c], acc);
  }
  return acc;
}

// tri[2e], tri[2e + 1] = the model at the 8 corners (bit 0: x + 1, bit 1:
// y + 1, bit 2: z + 1; 0 outside the grid) of base voxel e = (z0 + 1, y0 + 1,
// x0 + 1) over [-1, side)^3.
__global__ void tri_table_kernel(const float* __restrict__ model, int side, float4* tri) {
  const int64_t s1 = side + 1;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= s1 * s1 * s1) return;
  const int x0 = (int)(e % s1) - 1, y0 = (int)((e / s1) % s1) - 1, z0 = (int)(e / (s1 * s1)) - 1;
  float v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int kx = x0 + (c & 1), ky = y0 + ((c >> 1) & 1), kz = z0 + ((c >> 2) & 1);
    const bool in = kx >= 0 && kx < side && ky >= 0 && ky < side && kz >= 0 && kz < side;
    v[c] = in ? model[((int64_t)kz * side + ky) * side + kx] : 0.0f;
  }
  tri[2 * e] = make_float4(v[0], v[1], v[2], v[3]);
  tri[2 * e + 1] = make_float4(v[4], v[5], v[6], v[7]);
}

// The operand value of the split expansion and its FP16 hi / lo halves,
// packed hi | lo << 16.
__device__ __forceinline__ uint32_t split_bits(float w, float floor_, int log_split) {
  const float x = log_split ? logf(fmaxf(w, floor_)) : w;
  const __half hi = __float2half_rn(x);
  const __half lo = __float2half_rn(x - __half2float(hi));
  return (uint32_t)__half_as_ushort(hi) | ((uint32_t)__half_as_ushort(lo) << 16);
}

// The table's order, coordinates less one (voxels below 1 are never read):
// squares of 2 x 2 voxels in (y, z), 32 bytes each, along x, so a cache line
// holds 4 x 2 x 2 voxels.  A warp's pixels lie on a plane of any orientation and
// meet fewer sectors than with rows of voxels, which a plane across x meets
// one voxel at a time (86,520 rotations x 16,384 pixels: 3.9 -> 3.6 ms).
__host__ __device__ __forceinline__ int table_outside(int side) {
  return 4 * (side >> 1) * (side >> 1) * side;
}
__device__ __forceinline__ int table_entry(int x, int y, int z, int side) {
  // 4 ((z / 2 * (side / 2) + y / 2) * side + x) + 2 (z % 2) + y % 2
  const int row = 4 * side - 2, plane = 4 * (side >> 1) * side - 4;
  return (z >> 1) * plane + (y >> 1) * row + 4 * x + 2 * z + y;
}

template <int OUT>
__global__ void expand_table_kernel(const float* model, int side, float floor_, int log_split,
                                    uint2* tab) {
  auto value = [&](float w) {
    return OUT == EXP_LOG_F32 ? __float_as_uint(logf(fmaxf(w, floor_)))
                              : split_bits(w, floor_, log_split);
  };
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  const int M = side * side * side, end = table_outside(side);
  if (v >= M) {
    // a pixel outside the grid; a column past the last pixel
    if (v == M) tab[end] = make_uint2(0u, value(0.0f));
    if (v == M + 1) tab[end + 1] = make_uint2(0u, 0u);
    return;
  }
  const int q = v / side, x = v - q * side, z = q / side, y = q - z * side;
  if (x < 1 || y < 1 || z < 1) return;
  const float w = model[v];
  tab[table_entry(x - 1, y - 1, z - 1, side)] =
      make_uint2(__float_as_uint(w), value(w));
}

// A block expands `rot` <= 16 consecutive rotations over 256 pixels (of each of
// its `per` chunks of the detector): a thread keeps its two pixels' coordinates in
// registers and walks the rotations, four at a time, so eight gathers are in
// flight.  Consecutive rotations of the samplings are neighbours, so what one
// of them gathered for a compact patch of pixels (contexts list them along a
// Morton curve) is often in L1 for the next, and neither coordinates nor
// rotation matrices are loaded per pixel.  A block per rotation, as before,
// found 19% of its gathers in L1.  Nearest, through the table, is bound by the
// L1's sectors (97%) and nearly by its instructions (63 a pixel, 82%),
// trilinear by the L2 sector that each pixel takes:
//   86,520 rotations x 16,384 pixels, FP16 pair   5.0 -> 3.9, with the table's
//     order 3.6, with nearest_from_1 2.95 ms (5.7 GB written: 0.9 ms)
//   25,680 x 4,096  0.36 -> 0.29 -> 0.235 ms
//   25,680 x 12,800, FP32 logarithms 1.77 -> 1.38, with the table 0.98 ms
//
// Row statistics leave as one FP64 partial per (chunk group, rotation), summed
// in order by expand_rows_kernel, so they do not depend on the blocks' order.
constexpr int kExpThreads = 128, kExpChunk = 256, kExpRot = 16, kExpParts = 64;

// TAB: nearest, through the voxel table.
template <int INTERP, int OUT, bool TAB>
__global__ void __launch_bounds__(kExpThreads) expand_kernel(const ExpandArgs a, int rot,
                                                             int groups, int per) {
  __shared__ float4 ms[kExpRot][3];
  __shared__ double red[kExpThreads / 32][kExpRot];
  __shared__ uint32_t big[kExpThreads / 32][kExpRot];
  constexpr bool kHalf = OUT == EXP_F16_SPLIT;
  constexpr int kStep = INTERP == 0 ? 4 : 2;  // rotations in flight
  const int64_t rg = blockIdx.x / groups, r0 = rg * rot;
  const int cg = (int)(blockIdx.x - rg * groups);
  const int nr = (int)(a.R - r0 < rot ? a.R - r0 : rot);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < nr) {
    float m[9];
    emc_voxel::rotation_matrix(a.quat + 4 * (r0 + threadIdx.x), m);
    ms[threadIdx.x][0] = make_float4(m[0], m[1], m[2], 0.0f);
    ms[threadIdx.x][1] = make_float4(m[3], m[4], m[5], 0.0f);
    ms[threadIdx.x][2] = make_float4(m[6], m[7], m[8], 0.0f);
  }
  for (int k = lane; k < kExpRot; k += 32) {
    red[w][k] = 0.0;
    big[w][k] = 0;
  }
  __syncthreads();
  const int outside = table_outside(a.side);
  const int npix = (int)a.npix, ld = (int)a.ld;
  for (int c = cg * per; c < cg * per + per && c * kExpChunk < ld; ++c) {
    // two adjacent pixels (stored as half2), or two 128 apart (FP32 rows)
    int px[2];
    float x[2], y[2], z[2];
    int none[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      px[u] = c * kExpChunk + (kHalf ? 2 * threadIdx.x + u : threadIdx.x + u * kExpThreads);
      const bool in = px[u] < npix;
      // columns past the last pixel are outside the grid (and zero)
      x[u] = in ? a.cx[px[u]] : NAN;
      y[u] = in ? a.cy[px[u]] : NAN;
      z[u] = in ? a.cz[px[u]] : NAN;
      none[u] = outside + (in ? 0 : 1);
    }
#pragma unroll 1
    for (int k0 = 0; k0 < nr; k0 += kStep) {
      double st[kStep];
      uint32_t mx[kStep];
#pragma unroll
      for (int kk = 0; kk < kStep; ++kk) {
        const int k = k0 + kk;
        st[kk] = 0.0;
        mx[kk] = 0;
        if (k >= nr) continue;
        const float4 m0 = ms[k][0], m1 = ms[k][1], m2 = ms[k][2];
        const float m[9] = {m0.x, m0.y, m0.z, m1.x, m1.y, m1.z, m2.x, m2.y, m2.z};
        float v[2];
        uint32_t b[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          v[u] = 0.0f;
          b[u] = 0;
          float pos[3];
          if constexpr (TAB) {
            emc_voxel::position(m, a.side, x[u], y[u], z[u], pos);
            uint32_t e[3];
            const bool in = nearest_from_1(pos, a.side, e);
            const uint2 t = __ldg(a.tab + (in ? table_entry(e[0], e[1], e[2], a.side) : none[u]));
            v[u] = __uint_as_float(t.x);
            b[u] = t.y;
          } else {
            if (px[u] >= npix) continue;
            emc_voxel::position(m, a.side, x[u], y[u], z[u], pos);
            v[u] = (INTERP == 1 && a.tri) ? gather_tri(a.tri, pos, a.side)
                                          : gather<INTERP>(a.model, pos, a.side);
            if (kHalf)
              b[u] = split_bits(v[u], a.floor_, a.log_split);
            else
              b[u] = __float_as_uint(OUT == EXP_LOG_F32 ? logf(fmaxf(v[u], a.floor_)) : v[u]);
          }
        }
        if (a.stat != STAT_NONE)
          st[kk] = a.stat == STAT_SUMSQ ? (double)v[0] * v[0] + (double)v[1] * v[1]
                                        : (double)v[0] + (double)v[1];
        const int64_t row = (r0 + k) * a.ld;
        if constexpr (kHalf) {
          if (px[0] < ld) {  // ld is even
            *reinterpret_cast<uint32_t*>(a.out_hi + row + px[0]) = __byte_perm(b[0], b[1], 0x5410);
            *reinterpret_cast<uint32_t*>(a.out_lo + row + px[0]) = __byte_perm(b[0], b[1], 0x7632);
          }
        } else {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (px[u] >= ld) continue;
            const float o = __uint_as_float(b[u]);
            a.out_f32[row + px[u]] = o;
            mx[kk] = max(mx[kk], __float_as_uint(fabsf(o)));
          }
        }
      }
      if (a.stat != STAT_NONE) {
        // kStep row sums by halving exchanges
#pragma unroll
        for (int o = 16, n = kStep / 2; n >= 1; o >>= 1, n >>= 1) {
          const bool hi = lane & o;
#pragma unroll
          for (int q = 0; q < n; ++q) {
            const double keep = hi ? st[q + n] : st[q], send = hi ? st[q] : st[q + n];
            st[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        }
#pragma unroll
        for (int o = 16 / kStep; o > 0; o >>= 1) st[0] += __shfl_xor_sync(0xffffffffu, st[0], o);
        if (lane % (32 / kStep) == 0) red[w][k0 + lane / (32 / kStep)] += st[0];
      }
      if (!kHalf && a.rowmax) {
#pragma unroll
        for (int kk = 0; kk < kStep; ++kk) {
          const uint32_t q = __reduce_max_sync(0xffffffffu, mx[kk]);
          if (lane == 0) big[w][k0 + kk] = max(big[w][k0 + kk], q);
        }
      }
    }
  }
  if (a.stat == STAT_NONE && !a.rowmax) return;
  __syncthreads();
  if (threadIdx.x < nr) {
    double s = 0.0;
    uint32_t q = 0;
    for (int i = 0; i < kExpThreads / 32; ++i) {
      s += red[i][threadIdx.x];
      q = max(q, big[i][threadIdx.x]);
    }
    const int64_t o = (int64_t)cg * a.R + r0 + threadIdx.x;
    if (a.stat != STAT_NONE) a.statpart[o] = s;
    if (a.rowmax) a.maxpart[o] = __uint_as_float(q);
  }
}

__global__ void expand_rows_kernel(const ExpandArgs a, int groups) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= a.R) return;
  double s = 0.0;
  float mx = 0.0f;
  for (int g = 0; g < groups; ++g) {
    if (a.stat != STAT_NONE) s += a.statpart[g * a.R + r];
    if (a.rowmax) mx = fmaxf(mx, a.maxpart[g * a.R + r]);
  }
  if (a.stat != STAT_NONE) a.rowstat[r] = s;
  if (a.rowmax) a.rowmax[r] = mx;
}

__device__ __forceinline__ int64_t col_of(const int32_t* pix, int64_t j) { return pix ? pix[j] : j; }

// Likelihood: rows = rotations, columns = patterns, reduction over pixels.
struct OpLL {
  using Acc = double;
  static constexpr bool kBKMajor = true;
  LLArgs p;
  __device__ int64_t ksize() const { return p.npa; }
  __device__ float a(int64_t r, int64_t j) const {
    return (r < p.R && j < p.npa) ? __ldg(p.A + r * p.ldA + col_of(p.pix, j)) : 0.0f;
  }
  __device__ float b(int64_t n, int64_t j) const {
    if (n >= p.N || j >= p.npa) return 0.0f;
    const float k = __ldg(p.K + n * p.ldK + col_of(p.pix, j));
    return p.poisson ? k : k / __ldg(p.scaling + n);  // gaussian: image / scaling (emc_cuda.cu:121)
  }
  // inner(acc, a, b): each likelihood's own term, in OpLLGauss / OpLLPoisson
  __device__ void epilogue(double (&acc)[8][4], int64_t r0, int64_t n0, float*) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t r = r0 + i;
      if (r >= p.R) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t n = n0 + j;
        if (n >= p.N) continue;
        const double v = p.poisson ? acc[i][j] - (double)p.scaling[n] * p.rowstat[r]
                                   : -acc[i][j] * p.gauss_inv;
        if (p.LL64)
          p.LL64[r * p.ldLL + n] = v;
        else
          p.LL[r * p.ldLL + n] = (float)v;
      }
    }
  }
};
struct OpLLGauss : OpLL {
  static __device__ __forceinline__ float inner(float acc, float a, float b) {
    const float d = a - b;
    return fmaf(d, d, acc);
  }
};
struct OpLLPoisson : OpLL {
  static __device__ __forceinline__ float inner(float acc, float a, float b) { return fmaf(a, b, acc); }
};

// Gaussian scaling denominator: sum_r P_rp sum_j S_rj K_pj, reduced over the
// tile's rows in the epilogue.
struct OpCross {
  using Acc = float;
  static constexpr bool kBKMajor = true;
  CrossArgs p;
  __device__ int64_t ksize() const { return p.npa; }
  __device__ float a(int64_t r, int64_t j) const {
    return (r < p.R && j < p.npa) ? __ldg(p.S + r * p.ldS + col_of(p.pix, j)) : 0.0f;
  }
  __device__ float b(int64_t n, int64_t j) const {
    return (n < p.N && j < p.npa) ? __ldg(p.K + n * p.ldK + col_of(p.pix, j)) : 0.0f;
  }
  static __device__ __forceinline__ float inner(float acc, float a, float b) { return fmaf(a, b, acc); }
  __device__ void epilogue(float (&acc)[8][4], int64_t r0, int64_t n0, float* smem) const {
    double* red = reinterpret_cast<double*>(smem);  // [16][64]
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t n = n0 + j;
      double s = 0;
      if (n < p.N)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int64_t r = r0 + i;
          if (r < p.R) s += (double)__ldg(p.P + r * p.N + n) * acc[i][j];
        }
      red[ty * 64 + tx * 4 + j] = s;
    }
    __syncthreads();
    if (threadIdx.x < 64) {
      const int64_t n = (int64_t)blockIdx.x * TN + threadIdx.x;
      double s = 0;
      for (int k = 0; k < 16; ++k) s += red[k * 64 + threadIdx.x];
      if (n < p.N) p.den_part[(int64_t)blockIdx.y * p.N + n] = s;
    }
  }
};

// Slice average: rows = rotations, columns = pixels, reduction over patterns.
struct OpCompress {
  using Acc = float;
  static constexpr bool kBKMajor = false;
  CompressArgs p;
  __device__ int64_t ksize() const { return p.N; }
  __device__ float a(int64_t r, int64_t k) const {
    return (r < p.R && k < p.N) ? __ldg(p.P + r * p.N + k) : 0.0f;
  }
  __device__ float b(int64_t j, int64_t k) const {
    return (j < p.npa && k < p.N) ? __ldg(p.K + k * p.ldK + col_of(p.pix, j)) / __ldg(p.scaling + k)
                                  : 0.0f;
  }
  static __device__ __forceinline__ float inner(float acc, float a, float b) { return fmaf(a, b, acc); }
  __device__ void epilogue(float (&acc)[8][4], int64_t r0, int64_t j0, float*) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t r = r0 + i;
      if (r >= p.R) continue;
      const float T = p.T[r];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t jj = j0 + j;
        if (jj >= p.npa) continue;
        // emc_atomic.cu:105-111: divide by the slice's total responsibility
        p.U[r * p.ldU + col_of(p.pix, jj)] = T > 1e-30f ? acc[i][j] / T : acc[i][j];
      }
    }
  }
};

// ----------------------------------------------------------------- softmax --
// 32 patterns per block (lane == pattern), 8 warps share the rotations; X is
// the FP32 log-likelihood, overwritten by P in place (the drop-in API).
__global__ void __launch_bounds__(kBlock) softmax_kernel(float* X, int64_t R, int64_t N,
                                                         double* plogp_part, double* lse) {
  __shared__ float smax[8][32];
  __shared__ float ssum[8][32];
  __shared__ double sred[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t p = (int64_t)blockIdx.x * 32 + lane;
  const bool ok = p < N;
  float mx = -FLT_MAX;
  if (ok)
    for (int64_t r = w; r < R; r += 8) mx = X[r * N + p] > mx ? X[r * N + p] : mx;
  smax[w][lane] = mx;
  __syncthreads();
  mx = smax[0][lane];
  for (int k = 1; k < 8; ++k) mx = smax[k][lane] > mx ? smax[k][lane] : mx;
  float s = 0.0f;
  if (ok)
    for (int64_t r = w; r < R; r += 8) {
      const float d = X[r * N + p] - mx;
      if (d > -1.0e10f) s += expf(d);  // emc_cuda.cu:463-468
    }
  ssum[w][lane] = s;
  __syncthreads();
  s = 0.0f;
  for (int k = 0; k < 8; ++k) s += ssum[k][lane];
  const float inv = 1.0f / s;
  if (lse && ok && w == 0) lse[p] = (double)mx + log((double)s);
  double pl = 0.0;
  if (ok)
    for (int64_t r = w; r < R; r += 8) {
      const float d = X[r * N + p] - mx;
      const float P = d > -1.0e10f ? expf(d) * inv : 0.0f;
      X[r * N + p] = P;
      if (P > 0.0f) pl += (double)P * log((double)P);
    }
  sred[w][lane] = pl;
  __syncthreads();
  if (w == 0) {
    double t = 0;
    for (int k = 0; k < 8; ++k) t += sred[k][lane];
    t = warp_sum(t);
    if (lane == 0 && plogp_part) plogp_part[blockIdx.x] = t;
  }
}

// ------------------------------------ responsibilities of the FP32 contexts --
// Two sweeps over the FP64 log-likelihood, both bound by its HBM traffic.  One
// block walking every rotation of 32 patterns (63 blocks on 148 SMs at 2,000
// patterns) took 3.6 ms at 2,000 x 25,680 and 4.1 ms at 10,000 x 25,680; with
// the rotations split over blocks the two sweeps take 0.3 and 1.2 ms:
//   stats    per (row chunk, pattern) the online log-sum-exp and the sums the
//            scaling and sum P log P need, merged by resp_combine_kernel;
//   resp     P = exp(LL - lse), its row totals and row maxima.
// Exponentials are FP32 of FP64 differences; what is formed of them (the scaling's
// sum of P W or P C, sum P log P) is multiplied and summed in FP64.  FP32
// products folded four at a time took as long (10,000 x 25,680: 1.30 against
// 1.32 ms for the pass gaussian, 1.27 against 1.23 poisson, where weights of 0
// are skipped) and left the scaling an FP32 rounding further off.
// Rows in flight per warp.  Four, in 64 registers, leave room for a fourth block
// on an SM, which hides the sweep's loads better than eight in three blocks
// (45% of the issue slots): the pass of 10,000 x 25,680 1.38 -> 1.24 ms, 2,000 x
// 25,680 0.295 -> 0.272 ms.  Loading the next rows ahead: 1.27 to 1.36 ms.
constexpr int kStatRows = 4;

struct StatAcc {
  double m, s, d, q;  // max; sum e, sum e X, sum e (LL - m), e = exp(LL - m)
};
__device__ __forceinline__ void stat_rescale(StatAcc& a, double m) {
  if (m > a.m) {
    const double f = a.m > -DBL_MAX ? exp(a.m - m) : 0.0;
    a.q = f > 0.0 ? f * (a.q + (a.m - m) * a.s) : 0.0;
    a.s *= f;
    a.d *= f;
    a.m = m;
  }
}
__device__ __forceinline__ void stat_merge(StatAcc& a, const StatAcc& b) {
  if (b.m <= -DBL_MAX) return;
  stat_rescale(a, b.m);
  const double f = exp(b.m - a.m);
  a.q += f > 0.0 ? f * (b.q + (b.m - a.m) * b.s) : 0.0;
  a.s += f * b.s;
  a.d += f * b.d;
}

// The eight warps' sums of one pattern (lane), relative to their common
// maximum: one exponential per thread, the total on warp 0.  (The stats sweep
// merges them one after the other on warp 0 instead: with this reduction in it
// its main loop compiled to 1.14 instead of 0.74 ms at 10,000 x 25,680.)
__device__ __forceinline__ void stat_reduce(StatAcc& a, double (&sh)[4][8][32], int w, int lane) {
  sh[0][w][lane] = a.m;
  __syncthreads();
  double m = sh[0][0][lane];
#pragma unroll
  for (int k = 1; k < 8; ++k) m = fmax(m, sh[0][k][lane]);
  const double dm = a.m - m, f = a.m > -DBL_MAX ? exp(dm) : 0.0;
  sh[1][w][lane] = f * a.s;
  sh[2][w][lane] = f * a.d;
  sh[3][w][lane] = f > 0.0 ? f * (a.q + dm * a.s) : 0.0;
  __syncthreads();
  if (w != 0) return;
  a = StatAcc{m, 0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    a.s += sh[1][k][lane];
    a.d += sh[2][k][lane];
    a.q += sh[3][k][lane];
  }
}

template <bool POISSON>
__global__ void __launch_bounds__(256, 4) resp_stats_kernel(const RespF32Args a) {
  __shared__ double sh[8][32][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t cols = (a.N + 31) / 32, by = blockIdx.x / cols;
  const int64_t p = (blockIdx.x - by * cols) * 32 + lane;
  const bool ok = p < a.N;
  const int64_t r0 = by * a.chunk;
  const int64_t r1 = r0 + a.chunk < a.R ? r0 + a.chunk : a.R;
  // gaussian: X = sum S K from LL = (2 X / phi - sum S^2 - sum K^2 / phi^2) inv
  double half_phi = 0.0, k2 = 0.0, ginv = 0.0;
  if (!POISSON && ok) {
    const double phi = a.scaling[p];
    half_phi = 0.5 * phi;
    k2 = a.patstat[p] / (phi * phi);
    ginv = 1.0 / a.gauss_inv;
  }
  StatAcc acc{-DBL_MAX, 0.0, 0.0, 0.0};
  for (int64_t r = r0 + w * kStatRows; r < r1; r += 8 * kStatRows) {
    double v[kStatRows];
    double cm = -DBL_MAX;
#pragma unroll
    for (int k = 0; k < kStatRows; ++k)
      v[k] = ok && r + k < r1 ? a.LL[(r + k) * a.N + p] : -DBL_MAX;
#pragma unroll
    for (int k = 0; k < kStatRows; ++k) cm = v[k] > cm ? v[k] : cm;
    stat_rescale(acc, cm);
#pragma unroll
    for (int k = 0; k < kStatRows; ++k) {
      if (!(ok && r + k < r1)) continue;
      const double dl = v[k] - acc.m;
      const float e = expf(fmaxf((float)dl, -200.0f));
      if (!(e > 0.0f)) continue;  // also where LL is not finite
      const double rs = a.rowstat[r + k], x = POISSON ? rs : fma(v[k], ginv, rs + k2) * half_phi;
      acc.s += (double)e;
      acc.d = fma((double)e, x, acc.d);
      acc.q = fma((double)e, dl, acc.q);
    }
  }
  sh[w][lane][0] = acc.m;
  sh[w][lane][1] = acc.s;
  sh[w][lane][2] = acc.d;
  sh[w][lane][3] = acc.q;
  __syncthreads();
  if (w == 0 && ok) {
    for (int k = 1; k < 8; ++k)
      stat_merge(acc, StatAcc{sh[k][lane][0], sh[k][lane][1], sh[k][lane][2], sh[k][lane][3]});
    a.part[by * a.N + p] = make_double4(acc.m, acc.s, acc.d, acc.q);
  }
}

__global__ void __launch_bounds__(256) resp_combine_kernel(const RespF32Args a) {
  __shared__ double sh[4][8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t p = (int64_t)blockIdx.x * 32 + lane;
  const bool ok = p < a.N;
  StatAcc acc{-DBL_MAX, 0.0, 0.0, 0.0};
  if (ok) {
    for (int64_t k = w; k < a.nparts; k += 8) acc.m = fmax(acc.m, a.part[k * a.N + p].x);
    for (int64_t k = w; k < a.nparts; k += 8) {
      const double4 v = a.part[k * a.N + p];
      const double dm = v.x - acc.m, f = exp(dm);
      acc.s += f * v.y;
      acc.d += f * v.z;
      if (f > 0.0) acc.q += f * (v.w + dm * v.y);
    }
  }
  stat_reduce(acc, sh, w, lane);
  if (w != 0 || !ok) return;
  const double ls = log(acc.s);
  a.lse[p] = acc.m + ls;
  a.plogp[p] = acc.s > 0.0 ? acc.q / acc.s - ls : 0.0;  // sum P (LL - lse)
  // emc_cuda.cu:226; a pattern without photons or weight keeps its scale
  const double num = a.poisson ? a.patsum[p] : a.patstat[p], den = acc.d / acc.s;
  if (a.new_scaling) a.new_scaling[p] = num > 0.0 && den > 0.0 ? (float)(num / den) : a.scaling[p];
}

constexpr int kRespRows = 32, kRespStep = 8;

// 256 COLS patterns x `rows` rows per block, 8 rows at a time.  A thread sums its
// patterns' responsibilities first; the warp's 32 lanes are then reduced by
// halving exchanges (4 + 2 + 1 + 2 for 8 rows).  One pattern per thread, 16
// rows at a time and a division for the row maxima took 78 instructions an
// element and bound the sweep (73% of the issue slots).  The whole pass, with two
// patterns and the reciprocal: 10,000 x 25,680 1.50 -> 1.38 ms, 2,000 x 25,680
// 0.43 -> 0.30 ms; with four patterns, or 16 rows, there are fewer loads in
// flight (1.39 to 2.0 ms).
template <int COLS>
__global__ void __launch_bounds__(256) resp_kernel(const RespF32Args a, const int rows) {
  __shared__ double st[8][kRespRows];
  __shared__ uint32_t sm[8][kRespRows];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int kCols = 256 * COLS;
  const int64_t cols = (a.N + kCols - 1) / kCols, by = blockIdx.x / cols, bx = blockIdx.x - by * cols;
  double lse[COLS];
  float inv[COLS];  // the maxima may be one rounding off: launch_quant_rows has room for it
  int64_t p[COLS];
#pragma unroll
  for (int c = 0; c < COLS; ++c) {
    p[c] = bx * kCols + c * 256 + threadIdx.x;
    const bool ok = p[c] < a.N;
    lse[c] = ok ? a.lse[p[c]] : 0.0;
    inv[c] = ok ? 1.0f / (a.new_scaling ? a.new_scaling : a.scaling)[p[c]] : 0.0f;
  }
  const int64_t r0 = by * rows;
#pragma unroll 1
  for (int h = 0; h < rows; h += kRespStep) {
    double t[kRespStep];
    uint32_t b[kRespStep];
#pragma unroll
    for (int k = 0; k < kRespStep; ++k) {
      t[k] = 0.0;
      b[k] = 0;
    }
    double v[COLS][kRespStep];
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      const double* x = a.LL + (r0 + h) * a.N + p[c];
#pragma unroll
      for (int k = 0; k < kRespStep; ++k)
        v[c][k] = p[c] < a.N && r0 + h + k < a.R ? x[k * a.N] : -DBL_MAX;
    }
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      const bool ok = p[c] < a.N;
      float* y = a.P + (r0 + h) * a.N + p[c];
#pragma unroll
      for (int k = 0; k < kRespStep; ++k) {
        if (!(ok && r0 + h + k < a.R)) continue;
        // 0 also where LL or every LL of the pattern is not finite: the pattern
        // then takes no part (emc_cuda.cu:463-468 skips such terms)
        const float P = expf(fmaxf((float)(v[c][k] - lse[c]), -200.0f));
        y[k * a.N] = P;
        t[k] += (double)P;
        b[k] = max(b[k], __float_as_uint(P * inv[c]));  // >= 0; a NaN stays the largest
      }
    }
#pragma unroll
    for (int o = 16, n = kRespStep / 2; n >= 1; o >>= 1, n >>= 1) {
      const bool hi = lane & o;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const double keep = hi ? t[i + n] : t[i], send = hi ? t[i] : t[i + n];
        t[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        const uint32_t kb = hi ? b[i + n] : b[i], sb = hi ? b[i] : b[i + n];
        b[i] = max(kb, __shfl_xor_sync(0xffffffffu, sb, o));
      }
    }
#pragma unroll
    for (int o = 16 / kRespStep; o > 0; o >>= 1) {
      t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
      b[0] = max(b[0], __shfl_xor_sync(0xffffffffu, b[0], o));
    }
    if (lane % (32 / kRespStep) == 0) {
      st[w][h + lane / (32 / kRespStep)] = t[0];
      sm[w][h + lane / (32 / kRespStep)] = b[0];
    }
  }
  __syncthreads();
  if (threadIdx.x < rows && r0 + threadIdx.x < a.R) {
    double t = 0.0;
    uint32_t mx = 0;
    for (int k = 0; k < 8; ++k) {
      t += st[k][threadIdx.x];
      mx = max(mx, sm[k][threadIdx.x]);
    }
    a.Tpart[bx * a.R + r0 + threadIdx.x] = t;
    a.Mpart[bx * a.R + r0 + threadIdx.x] = __uint_as_float(mx);
  }
}

__global__ void resp_rows_kernel(const RespF32Args a, int64_t nblk) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= a.R) return;
  double t = 0.0;
  uint32_t mx = 0;
  for (int64_t b = 0; b < nblk; ++b) {
    t += a.Tpart[b * a.R + r];
    mx = max(mx, __float_as_uint(a.Mpart[b * a.R + r]));
  }
  a.T[r] = (float)t;
  a.rowmax[r] = __uint_as_float(mx);
  if (a.zero) a.zero[r] = 0;
}

__global__ void xlogx_partial(const float* x, int64_t n, double* part) {
  __shared__ double red[32];
  double s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float v = x[i];
    if (v > 0.0f) s += (double)v * log((double)v);
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// out[0] = sum of a, out[1] = sum of b: one block each.
__global__ void __launch_bounds__(1024) sum2_f64_kernel(const double* a, const double* b,
                                                        int64_t n, double* out) {
  __shared__ double red[32];
  const double* x = blockIdx.x ? b : a;
  double s = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += x[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

__global__ void sum_f64_kernel(const double* x, int64_t n, double* out) {
  __shared__ double red[32];
  double s = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += x[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) *out = s;
}

// --------------------------------------------------------------- scaling --
__global__ void scaling_finish_kernel(const double* num, const double* part, int64_t nparts,
                                      int64_t N, float* scaling) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  double d = 0;
  for (int64_t k = 0; k < nparts; ++k) d += part[k * N + p];
  // emc_cuda.cu:226; a pattern without photons or weight keeps its scale
  if (num[p] > 0.0 && d > 0.0) scaling[p] = (float)(num[p] / d);
}

__global__ void pattern_stats_kernel(const float* K, const int32_t* pix, int64_t N, int64_t npa,
                                     int64_t ldK, int squares, double* num) {
  const int64_t p = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= N) return;
  double s = 0;
  for (int64_t j = lane; j < npa; j += 32) {
    const double k = K[p * ldK + col_of(pix, j)];
    s += squares ? k * k : k;
  }
  s = warp_sum(s);
  if (lane == 0) num[p] = s;
}

// best[p] = argmax_r P[r][p] (first on ties), bestv[p] = that value: 32
// patterns per block (lane), the 8 warps split the rotations.
__global__ void __launch_bounds__(256) col_argmax_kernel(const float* P, int64_t R, int64_t N,
                                                         int32_t* best, float* bestv) {
  __shared__ float sv[8][32];
  __shared__ int32_t si[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t p = (int64_t)blockIdx.x * 32 + lane;
  float bv = -INFINITY;
  int32_t bi = -1;
  if (p < N)
    for (int64_t r = w; r < R; r += 8) {
      const float v = P[r * N + p];
      if (v > bv) {
        bv = v;
        bi = (int32_t)r;
      }
    }
  sv[w][lane] = bv;
  si[w][lane] = bi;
  __syncthreads();
  if (w == 0 && p < N) {
    for (int k = 1; k < 8; ++k)
      if (sv[k][lane] > bv || (sv[k][lane] == bv && si[k][lane] >= 0 && si[k][lane] < bi)) {
        bv = sv[k][lane];
        bi = si[k][lane];
      }
    best[p] = bi;
    bestv[p] = bv;
  }
}

__global__ void row_sums_kernel(const float* P, int64_t R, int64_t N, float* T) {
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= R) return;
  double s = 0;
  for (int64_t p = lane; p < N; p += 32) s += P[r * N + p];
  s = warp_sum(s);
  if (lane == 0) T[r] = (float)s;
}

// ----------------------------------------------------------------- insert --
// One block per rotation (emc_atomic.cu:115-133 + :17-73).
__global__ void __launch_bounds__(kBlock) insert_kernel(const InsertArgs a) {
  const int64_t r = blockIdx.x;
  const float T = a.T[r];
  // emc_atomic.cu:128 skips T_r <= 1e-10 (T_r over every pattern shard)
  if (!((a.Tskip ? a.Tskip[r] : T) > 1e-10f) || !(T > 0.0f)) return;
  const float w = a.rotw[r] * T;
  float m[9];
  emc_voxel::rotation_matrix(a.quat + 4 * r, m);
  for (int64_t i = threadIdx.x; i < a.npix; i += blockDim.x) {
    if (a.ins[i] != 1) continue;
    float u[3];
    emc_voxel::position(m, a.side, a.cx[i], a.cy[i], a.cz[i], u);
    const float s = a.U[r * a.ldU + i];
    // FP32 atomics, or the order-independent fixed-point limbs
    auto add = [&](int64_t v, float x, float y) {
      if (a.acc64) {
        add_fixed(a.acc64 + 8 * v, x);
        add_fixed(a.acc64 + 8 * v + 4, y);
      } else {
        atomicAdd(a.model + v, x);
        atomicAdd(a.weight + v, y);
      }
    };
    if (a.interp == 0) {
      int64_t v;
      if (!emc_voxel::nearest(u, a.side, 0, &v)) continue;
      add(v, w * s, w);
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        int64_t v;
        float wc;
        if (!emc_voxel::trilinear_corner(u, a.side, c, &v, &wc) || wc == 0.0f) continue;
        add(v, wc * w * s, wc * w);
      }
    }
  }
}

// The contexts' insertion of averaged slices U: interleaved (model, weight)
// pairs, so a voxel is one reduction instead of two, packed coordinates with
// four pixels in flight, and the trilinear corners by pairs (insert.cuh).
// With the slice sums before it: 10,000 patterns x 25,680 rotations at 64^3 4.14
// -> 3.74 ms, 2,000 x 25,680 at 128^3 4.04 -> 3.45 ms, 1,000 x 3,240 at 32^3 93
// -> 69 us.
template <int INTERP>
__global__ void __launch_bounds__(kBlock) insert_slices_kernel(const InsertArgs a) {
  constexpr int kUnroll = 4;
  const int64_t r = blockIdx.x;
  const float T = a.T[r];
  if (!((a.Tskip ? a.Tskip[r] : T) > 1e-10f) || !(T > 0.0f)) return;  // emc_atomic.cu:128
  const float w = a.rotw[r] * T;
  const InsertAcc to = acc_copy(a.to, r);
  float m[9];
  emc_voxel::rotation_matrix(a.quat + 4 * r, m);
  const float* U = a.U + r * a.ldU;
  const int n = (int)a.npix;
  for (int j0 = threadIdx.x; j0 < n; j0 += kUnroll * kBlock) {
    float4 q[kUnroll];
    float s[kUnroll];
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      const int j = j0 + k * kBlock;
      q[k] = j < n ? __ldg(a.pc + j) : make_float4(0.f, 0.f, 0.f, 0.f);
      s[k] = j < n ? U[j] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      if (q[k].w == 0.0f) continue;
      float u[3];
      emc_voxel::position(m, a.side, q[k].x, q[k].y, q[k].z, u);
      if constexpr (INTERP == 0)
        insert_nearest(to, u, a.side, w * s[k], w);
      else
        insert_trilinear(to, u, a.side, w * s[k], w);
    }
  }
}

// ------------------------------------------------------------- normalise --
// Fixed-point accumulators -> FP32 (value, weight) pairs: a[i*stride],
// b[i*stride] (the FP32 path's model and weight, or the mixed path's
// interleaved accumulators), each sum rounded once.
__global__ void fixed_to_pairs_kernel(const unsigned long long* acc64, int64_t M, float* a,
                                      float* b, int64_t stride) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (int64_t)gridDim.x * blockDim.x) {
    a[i * stride] = (float)fixed_value(acc64 + 8 * i);
    b[i * stride] = (float)fixed_value(acc64 + 8 * i + 4);
  }
}

// Both divisions also zero the counter the scaling after them finishes with.
__global__ void divide_kernel(float* model, const float* weight, int64_t M, int fp64,
                              double* part, unsigned int* done) {
  __shared__ double red[32];
  if (blockIdx.x == 0 && threadIdx.x == 0) *done = 0;
  double s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float wv = weight[i];
    float v;
    if (wv > 0.0f)  // emc_cuda.cu:416-420
      v = fp64 ? (float)((double)model[i] / (double)wv) : model[i] / wv;
    else
      v = 0.0f;
    model[i] = v;
    s += v;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// Mixed path: model/weight from the interleaved accumulators (FP64 division).
__global__ void divide_acc_kernel(const float2* acc, float* model, float* weight, int64_t M,
                                  double* part, unsigned int* done) {
  __shared__ double red[32];
  if (blockIdx.x == 0 && threadIdx.x == 0) *done = 0;
  double s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float2 a = acc[i];
    const float v = a.y > 0.0f ? (float)((double)a.x / (double)a.y) : 0.0f;  // emc_cuda.cu:416-420
    model[i] = v;
    weight[i] = a.y;
    s += v;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// model /= mean, its maximum to stats[1].  Every block sums the `nsum` partial
// sums of the division itself (the same order, so the same mean), and the last
// block to finish reduces the maxima, so no one-block kernel runs between the
// two sweeps or after them.  done[0] is 0 on entry and on exit.
__global__ void scale_max_kernel(float* model, int64_t M, const double* sums, int nsum, int fp64,
                                 double* stats, float* maxima, unsigned int* done) {
  __shared__ double red[32];
  __shared__ double total;
  __shared__ bool last;
  double s = 0.0;
  for (int i = threadIdx.x; i < nsum; i += blockDim.x) s += sums[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) total = s;
  __syncthreads();
  const double mean = total / (double)M;
  const float f = (float)(1.0 / mean);
  float mx = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (int64_t)gridDim.x * blockDim.x) {
    float v = model[i];
    if (mean != 0.0) v = fp64 ? (float)((double)v / mean) : v * f;
    model[i] = v;
    mx = fmaxf(mx, v);
  }
  mx = block_max(mx, reinterpret_cast<float*>(red));
  if (threadIdx.x == 0) {
    maxima[blockIdx.x] = mx;
    if (blockIdx.x == 0) stats[0] = mean;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  mx = 0.0f;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x)
    mx = fmaxf(mx, *reinterpret_cast<volatile float*>(maxima + i));
  mx = block_max(mx, reinterpret_cast<float*>(red));
  if (threadIdx.x == 0) {
    stats[1] = mx;
    *done = 0;
  }
}

__global__ void max_partial_kernel(const float* x, int64_t n, double* part) {
  __shared__ float red[32];
  float mx = -FLT_MAX;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    mx = fmaxf(mx, x[i]);
  mx = block_max(mx, red);
  if (threadIdx.x == 0) part[blockIdx.x] = mx;
}

__global__ void max_f64_kernel(const double* x, int64_t n, double* out) {
  __shared__ float red[32];
  float mx = -FLT_MAX;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) mx = fmaxf(mx, (float)x[i]);
  mx = block_max(mx, red);
  if (threadIdx.x == 0) *out = mx;
}

__global__ void fill_kernel(float* x, int64_t n, float v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] = v;
}

constexpr int kReduceBlocks = 592;  // 4 x 148 SMs; partial arrays hold this many values

inline int grid_for(int64_t n) {
  const int64_t b = (n + kBlock - 1) / kBlock;
  return (int)(b < kReduceBlocks ? (b > 0 ? b : 1) : kReduceBlocks);
}

}  // namespace

// ------------------------------------------------------------- launchers --

template <int INTERP, int OUT, bool TAB>
static void run_expand(const ExpandArgs& a, unsigned grid, int rot, int groups, int per,
                       cudaStream_t st) {
  expand_kernel<INTERP, OUT, TAB><<<grid, kExpThreads, 0, st>>>(a, rot, groups, per);
}

int64_t expand_parts(int64_t ld) {
  const int64_t chunks = (ld + kExpChunk - 1) / kExpChunk;
  return chunks < kExpParts ? chunks : kExpParts;
}

// Without the voxel table any side whose model fits the GPU; the table's index
// is 32 bits wide (contexts: side <= 1024).
cudaError_t launch_expand(const ExpandArgs& a, cudaStream_t st) {
  if (a.R <= 0) return cudaSuccess;
  if (a.npix > a.ld || a.ld > (int64_t)1 << 30 || a.side > 32768 || (a.tab && a.side > 1290) ||
      (a.out == EXP_F16_SPLIT && (a.ld % 2 != 0 || a.rowmax || (a.interp == 0 && !a.tab))) ||
      (a.stat != STAT_NONE && !(a.rowstat && a.statpart)) || (a.rowmax && !a.maxpart))
    return cudaErrorInvalidValue;
  const int64_t chunks = (a.ld + kExpChunk - 1) / kExpChunk;
  const int per = (int)((chunks + kExpParts - 1) / kExpParts);
  const int groups = (int)((chunks + per - 1) / per);
  // Fewer rotations a block where 16 would not give each SM four blocks: 1,000
  // rotations x 1,024 pixels is 252 blocks of 16, and one wave of them lasts as
  // long as 16 rotations take in a row.
  int rot = kExpRot;
  while (rot > 4 && groups * ((a.R + rot - 1) / rot) < 4 * 148) rot /= 2;
  const int64_t grid = groups * ((a.R + rot - 1) / rot);
  if (grid > 2147483647) return cudaErrorInvalidConfiguration;
  const bool near = a.interp == 0;
  auto run = a.out == EXP_F32       ? (near ? run_expand<0, EXP_F32, false> : run_expand<1, EXP_F32, false>)
             : a.out == EXP_LOG_F32 ? (!near   ? run_expand<1, EXP_LOG_F32, false>
                                       : a.tab ? run_expand<0, EXP_LOG_F32, true>
                                               : run_expand<0, EXP_LOG_F32, false>)
                                    : (near ? run_expand<0, EXP_F16_SPLIT, true>
                                            : run_expand<1, EXP_F16_SPLIT, false>);
  run(a, (unsigned)grid, rot, groups, per, st);
  if (a.stat != STAT_NONE || a.rowmax)
    expand_rows_kernel<<<(unsigned)((a.R + 255) / 256), 256, 0, st>>>(a, groups);
  return cudaGetLastError();
}

int64_t tri_table_entries(int side) { return 2 * (int64_t)(side + 1) * (side + 1) * (side + 1); }

cudaError_t launch_tri_table(const float* model, int side, float4* tri, cudaStream_t st) {
  const int64_t n = (int64_t)(side + 1) * (side + 1) * (side + 1);
  tri_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(model, side, tri);
  return cudaGetLastError();
}

int64_t expand_table_entries(int side) { return (int64_t)table_outside(side) + 2; }

cudaError_t launch_expand_table(const float* model, int side, int out, float floor_, int log_split,
                                uint2* tab, cudaStream_t st) {
  const int64_t M = (int64_t)side * side * side;
  if (out == EXP_LOG_F32)
    expand_table_kernel<EXP_LOG_F32><<<(unsigned)((M + 2 + 255) / 256), 256, 0, st>>>(
        model, side, floor_, log_split, tab);
  else
    expand_table_kernel<EXP_F16_SPLIT><<<(unsigned)((M + 2 + 255) / 256), 256, 0, st>>>(
        model, side, floor_, log_split, tab);
  return cudaGetLastError();
}

// ------------------------------------------------------------ photon lists --
// Gathers over the non-zero counts.  One block: 128 threads x 4 rotations =
// 512 rotations by 16 output columns (patterns of the log-likelihood, pixels
// of the slice sums).  For each column the block walks its entries (uniform
// loads of the sparse entry) and every thread gathers 16 bytes of the
// transposed operand row at that entry (logWT[pixel] for the log-likelihood,
// PT[pattern] for the slice sums), so one entry reads one coalesced 2 KB row.
// Column blocks vary fastest in the grid, so the blocks resident at one time
// share one rotation block's columns of the operand in L2.  FP32 partial sums
// over chunks of 32 entries are folded into FP64 totals, as the dense
// contraction folds each 32-wide K-step.  The 16 x 512 results leave through
// shared memory as rows of the output.
//   MODE 0: LL[r][p] = total - phi_p sum W_r      MODE 1: U[r][j] = total / T_r
constexpr int kSparseRot = 512, kSparsePat = 16;
template <int MODE>
__global__ void __launch_bounds__(128)
    sparse_gather_kernel(const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                         const float* __restrict__ val, const float* __restrict__ XT,
                         int64_t ldT, int64_t R, int64_t ncol, const float* scaling,
                         const double* rowstat, const float* T, float* out, double* out64) {
  __shared__ float tile[kSparsePat][kSparseRot + 1];
  const int64_t r0 = (int64_t)blockIdx.y * kSparseRot + 4 * threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * kSparsePat;
  const bool rv = r0 < R;  // ldT >= R rounded up to 4: the whole float4 is in bounds
  double sw[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (MODE == 0)
      sw[u] = r0 + u < R ? rowstat[r0 + u] : 0.0;
    else
      sw[u] = r0 + u < R ? (double)T[r0 + u] : 0.0;
  }
  for (int i = 0; i < kSparsePat; ++i) {
    const int64_t p = p0 + i;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (p < ncol && rv) {
      const int64_t e0 = ptr[p], e1 = ptr[p + 1];
      double tot[4] = {0.0, 0.0, 0.0, 0.0};
      int64_t e = e0;
      while (e < e1) {
        const int64_t ce = e + 32 < e1 ? e + 32 : e1;
        float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
        for (; e + 2 <= ce; e += 2) {
          const int32_t j0 = __ldg(idx + e), j1 = __ldg(idx + e + 1);
          const float k0 = __ldg(val + e), k1 = __ldg(val + e + 1);
          const float4 w0 = __ldg(reinterpret_cast<const float4*>(XT + (int64_t)j0 * ldT + r0));
          const float4 w1 = __ldg(reinterpret_cast<const float4*>(XT + (int64_t)j1 * ldT + r0));
          s0.x = fmaf(k0, w0.x, s0.x); s0.y = fmaf(k0, w0.y, s0.y);
          s0.z = fmaf(k0, w0.z, s0.z); s0.w = fmaf(k0, w0.w, s0.w);
          s1.x = fmaf(k1, w1.x, s1.x); s1.y = fmaf(k1, w1.y, s1.y);
          s1.z = fmaf(k1, w1.z, s1.z); s1.w = fmaf(k1, w1.w, s1.w);
        }
        if (e < ce) {
          const float k0 = __ldg(val + e);
          const float4 w0 =
              __ldg(reinterpret_cast<const float4*>(XT + (int64_t)__ldg(idx + e) * ldT + r0));
          s0.x = fmaf(k0, w0.x, s0.x); s0.y = fmaf(k0, w0.y, s0.y);
          s0.z = fmaf(k0, w0.z, s0.z); s0.w = fmaf(k0, w0.w, s0.w);
          ++e;
        }
        tot[0] += (double)(s0.x + s1.x);
        tot[1] += (double)(s0.y + s1.y);
        tot[2] += (double)(s0.z + s1.z);
        tot[3] += (double)(s0.w + s1.w);
      }
      if (MODE == 0) {
        const double ph = (double)scaling[p];
        if (out64) {
          // FP64 results leave from registers (one column of 4 rows each)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (r0 + u < R) out64[(r0 + u) * ncol + p] = tot[u] - ph * sw[u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = (float)(tot[u] - ph * sw[u]);
      } else {
        // emc_atomic.cu:105-111: divide by the slice's total responsibility
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float Tr = (float)sw[u];
          v[u] = Tr > 1e-30f ? (float)tot[u] / Tr : (float)tot[u];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) tile[i][4 * threadIdx.x + u] = v[u];
  }
  if (out64) return;  // uniform over the block
  __syncthreads();
  // half a warp per output row: lane & 15 = column
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t p = p0 + (lane & 15);
  for (int rr = 2 * w + (lane >> 4); rr < kSparseRot; rr += 8) {
    const int64_t ro = (int64_t)blockIdx.y * kSparseRot + rr;
    if (ro < R && p < ncol) out[ro * ncol + p] = tile[lane & 15][rr];
  }
}

__global__ void scale_entries_kernel(const float* val, const int32_t* row, const float* scaling,
                                     int64_t nnz, float* out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < nnz) out[e] = val[e] / scaling[row[e]];
}

cudaError_t launch_ll_sparse(const SparseLLArgs& a, cudaStream_t st) {
  if (a.R <= 0 || a.N <= 0) return cudaSuccess;
  if (a.ldT % 4 != 0 || a.ldT < a.R || (reinterpret_cast<uintptr_t>(a.logWT) & 15u))
    return cudaErrorInvalidValue;
  dim3 grid((unsigned)((a.N + kSparsePat - 1) / kSparsePat),
            (unsigned)((a.R + kSparseRot - 1) / kSparseRot));
  if (grid.y > 65535u) return cudaErrorInvalidConfiguration;
  sparse_gather_kernel<0><<<grid, 128, 0, st>>>(a.row_ptr, a.col, a.val, a.logWT, a.ldT, a.R, a.N,
                                                a.scaling, a.rowstat, nullptr, a.LL, a.LL64);
  return cudaGetLastError();
}

cudaError_t launch_compress_sparse(const SparseCmpArgs& a, cudaStream_t st) {
  if (a.R <= 0 || a.npa <= 0) return cudaSuccess;
  if (a.ldT % 4 != 0 || a.ldT < a.R || (reinterpret_cast<uintptr_t>(a.PT) & 15u))
    return cudaErrorInvalidValue;
  dim3 grid((unsigned)((a.npa + kSparsePat - 1) / kSparsePat),
            (unsigned)((a.R + kSparseRot - 1) / kSparseRot));
  if (grid.y > 65535u) return cudaErrorInvalidConfiguration;
  sparse_gather_kernel<1><<<grid, 128, 0, st>>>(a.col_ptr, a.row, a.val, a.PT, a.ldT, a.R, a.npa,
                                                nullptr, nullptr, a.T, a.U, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_scale_entries(const float* val, const int32_t* row, const float* scaling,
                                 int64_t nnz, float* val_out, cudaStream_t st) {
  if (nnz <= 0) return cudaSuccess;
  scale_entries_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, st>>>(val, row, scaling, nnz,
                                                                     val_out);
  return cudaGetLastError();
}

__global__ void transpose_kernel(const float* S, int64_t R, int64_t npa, float* ST, int64_t ldT) {
  __shared__ float t[32][33];
  const int64_t j0 = (int64_t)blockIdx.x * 32, r0 = (int64_t)blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int64_t r = r0 + i, j = j0 + threadIdx.x;
    t[i][threadIdx.x] = (r < R && j < npa) ? S[r * npa + j] : 0.0f;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += 8) {
    const int64_t j = j0 + i, r = r0 + threadIdx.x;
    if (j < npa && r < R) ST[j * ldT + r] = t[threadIdx.x][i];
  }
}

cudaError_t launch_transpose(const float* S, int64_t R, int64_t npa, float* ST, int64_t ldT,
                             cudaStream_t st) {
  dim3 grid((unsigned)((npa + 31) / 32), (unsigned)((R + 31) / 32));
  if (grid.y > 65535u) return cudaErrorInvalidConfiguration;
  transpose_kernel<<<grid, dim3(32, 8), 0, st>>>(S, R, npa, ST, ldT);
  return cudaGetLastError();
}

// one warp per pattern
__global__ void csr_count_kernel(const float* K, int64_t N, int64_t npa, int64_t* count) {
  const int64_t p = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= N) return;
  int64_t n = 0;
  for (int64_t j = lane; j < npa; j += 32) n += K[p * npa + j] != 0.0f;
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if (lane == 0) count[p] = n;
}

__global__ void csr_fill_kernel(const float* K, int64_t N, int64_t npa, const int64_t* row_ptr,
                                int32_t* col, float* val) {
  const int64_t p = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= N) return;
  int64_t out = row_ptr[p];
  for (int64_t j0 = 0; j0 < npa; j0 += 32) {
    const int64_t j = j0 + lane;
    const float k = j < npa ? K[p * npa + j] : 0.0f;
    const unsigned nz = __ballot_sync(0xffffffffu, k != 0.0f);
    if (k != 0.0f) {
      const int64_t o = out + __popc(nz & ((1u << lane) - 1u));
      col[o] = (int32_t)j;
      val[o] = k;
    }
    out += __popc(nz);
  }
}

cudaError_t launch_csr_count(const float* K, int64_t N, int64_t npa, int64_t* count,
                             cudaStream_t st) {
  csr_count_kernel<<<(unsigned)((N + 7) / 8), 256, 0, st>>>(K, N, npa, count);
  return cudaGetLastError();
}

cudaError_t launch_csr_fill(const float* K, int64_t N, int64_t npa, const int64_t* row_ptr,
                            int32_t* col, float* val, cudaStream_t st) {
  csr_fill_kernel<<<(unsigned)((N + 7) / 8), 256, 0, st>>>(K, N, npa, row_ptr, col, val);
  return cudaGetLastError();
}

cudaError_t launch_ll_fp32(const LLArgs& a, cudaStream_t st) {
  if (a.R <= 0 || a.N <= 0) return cudaSuccess;
  dim3 grid((unsigned)((a.N + TN - 1) / TN), (unsigned)((a.R + TM - 1) / TM));
  if (a.poisson) {
    OpLLPoisson op;
    op.p = a;
    tile_kernel<<<grid, kBlock, 0, st>>>(op);
  } else {
    OpLLGauss op;
    op.p = a;
    tile_kernel<<<grid, kBlock, 0, st>>>(op);
  }
  return cudaGetLastError();
}

int64_t resp_f32_blocks(int64_t N) { return (N + 255) / 256; }

// Rows per block of the stats sweep: at least 64 (eight per warp),
// more where the patterns alone fill the GPU several times.
int64_t resp_f32_chunk(int64_t R, int64_t N) {
  const int64_t cols = (N + 31) / 32, want = 8 * 148;  // blocks
  int64_t parts = (want + cols - 1) / cols;
  const int64_t most = (R + 63) / 64;
  if (parts > most) parts = most;
  int64_t chunk = (R + parts - 1) / parts;
  if (chunk > 2048) chunk = 2048;
  return (chunk + 63) / 64 * 64;
}

cudaError_t launch_resp_f32(const RespF32Args& a, cudaStream_t st) {
  const int64_t cols = (a.N + 31) / 32;
  const unsigned gs = (unsigned)(cols * a.nparts);
  if (a.poisson)
    resp_stats_kernel<true><<<gs, 256, 0, st>>>(a);
  else
    resp_stats_kernel<false><<<gs, 256, 0, st>>>(a);
  resp_combine_kernel<<<(unsigned)cols, 256, 0, st>>>(a);
  // two patterns a thread, one (then fewer rows a block) where that would not
  // give each SM eight blocks (four): 1,000 x 3,240 is 204 blocks, the pass 58
  // -> 52 us with one pattern, and 64 x 420 34 -> 28 us with 8 rows
  int rows = kRespRows, c = 2;
  auto blocks = [&](int c, int rows) {
    return ((a.N + 256 * c - 1) / (256 * c)) * ((a.R + rows - 1) / rows);
  };
  if (blocks(c, rows) < 8 * 148) c = 1;
  while (rows > kRespStep && blocks(c, rows) < 4 * 148) rows /= 2;
  const int64_t nb = (a.N + 256 * c - 1) / (256 * c);
  auto run = c == 2 ? resp_kernel<2> : resp_kernel<1>;
  run<<<(unsigned)blocks(c, rows), 256, 0, st>>>(a, rows);
  resp_rows_kernel<<<(unsigned)((a.R + 255) / 256), 256, 0, st>>>(a, nb);
  return cudaGetLastError();
}

cudaError_t launch_softmax_fp32(float* X, int64_t R, int64_t N, double* plogp_part, int* nparts,
                                double* lse, cudaStream_t st) {
  const int64_t nb = (N + 31) / 32;
  if (nparts) *nparts = (int)nb;
  softmax_kernel<<<(unsigned)nb, kBlock, 0, st>>>(X, R, N, plogp_part, lse);
  return cudaGetLastError();
}

cudaError_t launch_xlogx_sum(const float* x, int64_t n, double* out, double* scratch,
                             cudaStream_t st) {
  const int g = grid_for(n);
  xlogx_partial<<<g, kBlock, 0, st>>>(x, n, scratch);
  sum_f64_kernel<<<1, kBlock, 0, st>>>(scratch, g, out);
  return cudaGetLastError();
}

cudaError_t launch_scaling_cross(const CrossArgs& a, cudaStream_t st) {
  dim3 grid((unsigned)((a.N + TN - 1) / TN), (unsigned)((a.R + TM - 1) / TM));
  OpCross op;
  op.p = a;
  tile_kernel<<<grid, kBlock, 0, st>>>(op);
  return cudaGetLastError();
}

cudaError_t launch_scaling_finish(const double* num, const double* den_part, int64_t nparts,
                                  int64_t N, float* scaling, cudaStream_t st) {
  scaling_finish_kernel<<<(unsigned)((N + kBlock - 1) / kBlock), kBlock, 0, st>>>(num, den_part,
                                                                                 nparts, N, scaling);
  return cudaGetLastError();
}

cudaError_t launch_pattern_stats(const float* K, const int32_t* pix, int64_t N, int64_t npa,
                                 int64_t ldK, int squares, double* num, cudaStream_t st) {
  pattern_stats_kernel<<<(unsigned)((N + 7) / 8), kBlock, 0, st>>>(K, pix, N, npa, ldK, squares, num);
  return cudaGetLastError();
}

cudaError_t launch_col_argmax(const float* P, int64_t R, int64_t N, int32_t* best, float* bestv,
                              cudaStream_t st) {
  col_argmax_kernel<<<(unsigned)((N + 31) / 32), 256, 0, st>>>(P, R, N, best, bestv);
  return cudaGetLastError();
}

cudaError_t launch_row_sums(const float* P, int64_t R, int64_t N, float* T, cudaStream_t st) {
  row_sums_kernel<<<(unsigned)((R + 7) / 8), kBlock, 0, st>>>(P, R, N, T);
  return cudaGetLastError();
}

cudaError_t launch_compress_fp32(const CompressArgs& a, cudaStream_t st) {
  dim3 grid((unsigned)((a.npa + TN - 1) / TN), (unsigned)((a.R + TM - 1) / TM));
  OpCompress op;
  op.p = a;
  tile_kernel<<<grid, kBlock, 0, st>>>(op);
  return cudaGetLastError();
}

cudaError_t launch_insert(const InsertArgs& a, cudaStream_t st) {
  if (a.R <= 0) return cudaSuccess;
  if (a.pc && a.interp == 0)
    insert_slices_kernel<0><<<(unsigned)a.R, kBlock, 0, st>>>(a);
  else if (a.pc)
    insert_slices_kernel<1><<<(unsigned)a.R, kBlock, 0, st>>>(a);
  else
    insert_kernel<<<(unsigned)a.R, kBlock, 0, st>>>(a);
  return cudaGetLastError();
}

// Scratch of a normalisation (kReduceBlocks + kReduceBlocks / 2 + 1 doubles):
// partial sums, block maxima, the counter of finished blocks.
static void scale_after_division(float* model, int64_t M, int g, int fp64, double* scratch,
                                 double* stats, cudaStream_t st) {
  float* maxima = reinterpret_cast<float*>(scratch + kReduceBlocks);
  unsigned int* done = reinterpret_cast<unsigned int*>(maxima + kReduceBlocks);
  scale_max_kernel<<<g, kBlock, 0, st>>>(model, M, scratch, g, fp64, stats, maxima, done);
}
static unsigned int* done_counter(double* scratch) {
  return reinterpret_cast<unsigned int*>(scratch + kReduceBlocks) + kReduceBlocks;
}

cudaError_t launch_normalize_model(float* model, const float* weight, int64_t M, int fp64,
                                   double* scratch, double* stats, cudaStream_t st) {
  // stats[0] = mean, stats[1] = max
  const int g = grid_for(M);
  divide_kernel<<<g, kBlock, 0, st>>>(model, weight, M, fp64, scratch, done_counter(scratch));
  scale_after_division(model, M, g, fp64, scratch, stats, st);
  return cudaGetLastError();
}

cudaError_t launch_fixed_to_pairs(const unsigned long long* acc64, int64_t M, float* a, float* b,
                                  int64_t stride, cudaStream_t st) {
  fixed_to_pairs_kernel<<<grid_for(M), kBlock, 0, st>>>(acc64, M, a, b, stride);
  return cudaGetLastError();
}

cudaError_t launch_normalize_acc(const float2* acc, float* model, float* weight, int64_t M,
                                 double* scratch, double* stats, cudaStream_t st) {
  const int g = grid_for(M);
  divide_acc_kernel<<<g, kBlock, 0, st>>>(acc, model, weight, M, scratch, done_counter(scratch));
  scale_after_division(model, M, g, 1, scratch, stats, st);
  return cudaGetLastError();
}

cudaError_t launch_model_max(const float* model, int64_t M, double* scratch, double* out,
                             cudaStream_t st) {
  const int g = grid_for(M);
  max_partial_kernel<<<g, kBlock, 0, st>>>(model, M, scratch);
  max_f64_kernel<<<1, kBlock, 0, st>>>(scratch, g, out);
  return cudaGetLastError();
}

cudaError_t launch_fill(float* x, int64_t n, float v, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  fill_kernel<<<grid_for(n), kBlock, 0, st>>>(x, n, v);
  return cudaGetLastError();
}

cudaError_t launch_sum2_f64(const double* a, const double* b, int64_t n, double* out,
                            cudaStream_t st) {
  sum2_f64_kernel<<<2, 1024, 0, st>>>(a, b, n, out);
  return cudaGetLastError();
}

cudaError_t launch_sum_f64(const double* x, int64_t n, double* out, cudaStream_t st) {
  sum_f64_kernel<<<1, kBlock, 0, st>>>(x, n, out);
  return cudaGetLastError();
}

}  // namespace emc
