// FP32 contractions of the context API on the tensor cores, exact by
// construction: out[n][m] = sum_k A[m][k] X[n][k] with A small integers (photon
// counts) and X FP32 (slices, log slices, responsibilities).
//
// Each row of X becomes a fixed-point integer per element, 30 bits and sign
// relative to the row's largest magnitude (a power-of-two unit, so every
// element within 2^-7 of it keeps all its FP32 bits), cut into four balanced
// base-256 digits; the counts are signed bytes (0 .. 127, or base-128 digits
// in two passes).  tcgen05.mma kind::i8 multiplies the bytes and accumulates
// in 32-bit integers, one TMEM accumulator per digit, and the epilogue
// recombines the four sums as one 64-bit integer: no rounding happens between
// the quantisation and the final conversion to FP64.  The quantisation error is
// absolute, 2^-31 of the row maximum per element.  For the log-likelihood, a sum
// over the same row, that is below the rounding of the FP32 partial sums it
// replaces.  The slice sums need relative precision: a pixel may have photons
// only from patterns whose responsibility is far below the row's largest.  Where a
// sum is so small that the fixed point shows, small_terms_kernel adds what it
// left out.
//
// What bounds it: the tensor pipe; four byte digits cost the MMA time of two
// FP16 operand halves.  Measured (10,000 patterns x 25,680 rotations x 4,044
// pixels): 3.2 ms, 646 TFLOP/s of the contraction, where the register-tiled
// CUDA-core form, held by its shared-memory loads and FP64 folds, takes 92 to
// 255 ms; 2,000 x 25,680 x 16,272: 2.4 against 92 ms.  SM pairs (cta_group::2) compute 256 x 128 tiles: 128 columns,
// since the four digit accumulators fill the 512 TMEM columns; TMEM then has
// no second buffer, so sixteen epilogue warps first drain the accumulators
// into registers (32 columns each, recombined to 64 bits as they come) and
// release them, and convert and store behind the next tile's MMAs.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "i8.cuh"
#include "tc_ptx.cuh"

namespace emc {
namespace {

constexpr int kTileM = 256, kTileN = 128;  // of an SM pair
constexpr int kStepK = 128;                // bytes per shared-memory row and K-step
constexpr int kStages = 4;
constexpr int kDigits = kI8Digits;
constexpr int kEpiWarps = 16;
constexpr int kEpiThreads = 32 * kEpiWarps;
constexpr int kWarpCols = kTileN / (kEpiWarps / 4);  // columns per epilogue warp
constexpr uint32_t kABytes = 128 * kStepK;               // this CTA's 128 rows of A
constexpr uint32_t kBBytes = (kTileN / 2) * kStepK;      // its half of one digit plane
constexpr uint32_t kStageBytes = kABytes + kDigits * kBBytes;
// kind::i8, D = S32, A = B = S8 (both K-major), N = 128, M = 256 over the pair
constexpr uint32_t kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) |
                              ((uint32_t)(kTileN >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);

__device__ __forceinline__ void mma_i8_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(kIdescI8), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&v)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7])
      : "r"(taddr));
}

// Column constants of a tile in shared memory (two tiles' worth: the stores
// of one tile run while the next one's constants arrive).
struct ColConst {
  double unit;  // value of one unit of the column's integer sum
  double c;     // per-column term of the epilogue
  float few;    // slice sums: kSmallUnits units
};

// LL[n][m], n = rotation, m = pattern:
//   poisson   C - phi sum W            gaussian  (2 C / phi - sum S^2 - sum K^2 / phi^2) inv
struct EpiLL {
  I8LLArgs a;
  double c1, c0;
  __device__ void column(int64_t n, ColConst& k) const {
    const bool ok = n < a.R;
    k.unit = ok ? (double)a.unit[n] * a.mult : 0.0;
    k.c = ok ? (a.poisson ? a.rowstat[n] : a.rowstat[n] * a.gauss_inv) : 0.0;
  }
  __device__ void row(int64_t m) {
    c1 = c0 = 0.0;
    if (m >= a.N) return;
    const double phi = a.scaling[m];
    if (a.poisson) {
      c1 = phi;
    } else {
      c1 = 2.0 * a.gauss_inv / phi;
      c0 = -a.patstat[m] / (phi * phi) * a.gauss_inv;
    }
  }
  __device__ void store(int64_t m, int64_t n, long long v, const ColConst& k) const {
    if (m >= a.N || n >= a.R) return;
    double* o = a.LL + n * a.N + m;
    double x = (double)v * k.unit;
    if (a.pass == I8_HIGH) {  // the base-128 digit of the counts: the bare sum
      *o = x;
      return;
    }
    if (a.pass == I8_LOW) x += *o;
    *o = a.poisson ? fma(-c1, k.c, x) : fma(x, c1, c0 - k.c);
  }
  __device__ void stored(int64_t, int) {}
};

// U[n][m] = sum / T_n, n = rotation, m = active pixel (emc_atomic.cu:105-111).
// A term is off by half a unit at most, so a sum of at least kSmallUnits units
// per photon at the pixel is within 2^-21, and within that over the root of the
// number of terms where the errors are independent.  Rows with a smaller sum are
// flagged: none of them with broad posteriors (10,000 patterns x 25,680 rotations
// gaussian), nearly all with sharp ones.
constexpr float kSmallUnits = 1048576.0f;
struct EpiU {
  I8UArgs a;
  float kt;
  uint32_t small = 0;
  __device__ void column(int64_t n, ColConst& k) const {
    const bool ok = n < a.R;
    const float T = ok ? a.T[n] : 1.0f;
    const double u = ok ? (double)a.unit[n] / (T > 1e-30f ? (double)T : 1.0) : 0.0;
    k.unit = u * a.mult;
    k.c = 0.0;
    k.few = (float)u * kSmallUnits;
  }
  __device__ void row(int64_t m) { kt = m < a.npa ? (float)a.ktot[m] : 0.0f; }
  __device__ void store(int64_t m, int64_t n, long long v, const ColConst& k) {
    if (m >= a.npa || n >= a.R) return;
    float* o = a.U + n * a.npa + m;
    double x = (double)v * k.unit;
    if (a.pass == I8_LOW) x += (double)*o;
    const float y = (float)x;
    *o = y;
    if (y <= kt * k.few) small |= 1u << (n & 31);
  }
  // One store of 32 flags per warp: every SM is at the same rows, and a store per
  // element to them took longer than the contraction.
  __device__ void stored(int64_t n0, int lane) {
    const uint32_t b = __reduce_or_sync(0xffffffffu, kt > 0.0f ? small : 0u);
    if (a.pass != I8_HIGH && n0 + lane < a.R && (b >> lane & 1u)) a.flag[n0 + lane] = 1;
    small = 0;
  }
};
static_assert(kWarpCols == 32, "EpiU keeps a bit per column");

template <class Epi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + kEpiThreads, 1)
    i8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const int64_t m_tiles, const int64_t n_tiles, const int64_t k_blocks,
                   const int64_t plane_rows, const Epi epi, TcStatus* status) {
  extern __shared__ uint8_t dyn_smem[];
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages];
  __shared__ __align__(8) uint64_t tfull_bar, tempty_bar, drain_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, epi_abort;
  __shared__ ColConst cols[2][kTileN];

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) &
                                             ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  Ctl ctl{&abort_flag, status};
  auto abort_pair = [&]() {  // the peer's waits end at their next check too
    abort_flag = 1;
    const uint32_t pa = peer_addr(smem_u32(&abort_flag), rank ^ 1u);
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(pa), "r"(1) : "memory");
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(&tfull_bar), 1);
    mbar_init(smem_u32(&tempty_bar), 2);  // one arrival per CTA's epilogue
    mbar_init(smem_u32(&drain_bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(kDigits * kTileN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const int64_t num_tiles = m_tiles * n_tiles;
  const int64_t cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;

  // m fastest: the SMs in flight share the digit tiles (bands of n tiles: no change)
  auto tile_mn = [&](int64_t t, int64_t& m, int64_t& n) {
    n = t / m_tiles;
    m = t - n * m_tiles;
  };

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------ TMA producer (both CTAs)
      int s = 0;
      uint32_t ph = 0;
      int64_t issued = 0;
      bool ok = true;
      for (int64_t t = cid; t < num_tiles && ok; t += ncl) {
        int64_t mt, nt;
        tile_mn(t, mt, nt);
        const int ar = (int)(mt * kTileM + rank * 128);
        const int br = (int)(nt * kTileN + rank * (kTileN / 2));
        for (int64_t kb = 0; kb < k_blocks; ++kb) {
          if (!bounded_wait(smem_u32(&empty_bar[s]), ph ^ 1, ctl, 11)) {
            ok = false;
            break;
          }
          const uint32_t fb = smem_u32(&full_bar[s]);
          if (leader) mbar_expect_tx(fb, 2 * kStageBytes);  // both CTAs' bytes
          const uint32_t fb_leader = peer_addr(fb, 0);
          const uint32_t base = smem_u32(smem + (size_t)s * kStageBytes);
          const int kc = (int)(kb * kStepK);
          tma_load_2d_pair(base, &tmA, kc, ar, fb_leader);
#pragma unroll
          for (int q = 0; q < kDigits; ++q)
            tma_load_2d_pair(base + kABytes + q * kBBytes, &tmB, kc, br + (int)(q * plane_rows),
                             fb_leader);
          ++issued;
          if (++s == kStages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (!ok) {
        abort_pair();
        if (leader) {
          // the last min(issued, stages) stages must land (both CTAs' bytes
          // complete on these barriers) before the pair exits
          const int64_t n = issued < kStages ? issued : kStages;
          int ss = s;
          uint32_t pp = ph;
          for (int64_t i = 0; i < n; ++i) {
            if (--ss < 0) {
              ss = kStages - 1;
              pp ^= 1;
            }
            const uint64_t t0 = globaltimer();
            while (!mbar_test(smem_u32(&full_bar[ss]), pp) && globaltimer() - t0 < kWaitLimitNs) {
            }
          }
        } else {
          // the peer cannot observe its loads; give them time to land
          const uint64_t t0 = globaltimer();
          while (globaltimer() - t0 < 2000000ull) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {
      // ------------------------------------------------ MMA issuer (leader)
      int s = 0;
      uint32_t ph = 0, i = 0;
      bool ok = true;
      for (int64_t t = cid; t < num_tiles && ok; t += ncl, ++i) {
        if (!bounded_wait(smem_u32(&tempty_bar), (i & 1) ^ 1, ctl, 12)) {
          abort_pair();
          break;
        }
        tc_fence_after();
        for (int64_t kb = 0; kb < k_blocks; ++kb) {
          if (!bounded_wait(smem_u32(&full_bar[s]), ph, ctl, 13)) {
            ok = false;
            abort_pair();
            break;
          }
          tc_fence_after();
          const uint32_t base = smem_u32(smem + (size_t)s * kStageBytes);
#pragma unroll
          for (int k = 0; k < kStepK / 32; ++k)
#pragma unroll
            for (int q = 0; q < kDigits; ++q)
              mma_i8_pair(tmem + q * kTileN, sdesc<64>(base + k * 32),
                          sdesc<64>(base + kABytes + q * kBBytes + k * 32), (kb | k) != 0);
          const uint32_t eb = smem_u32(&empty_bar[s]);
          mma_commit_pair(peer_addr(eb, 0));
          mma_commit_pair(peer_addr(eb, 1));
          if (++s == kStages) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok) {
          const uint32_t tb = smem_u32(&tfull_bar);
          mma_commit_pair(peer_addr(tb, 0));
          mma_commit_pair(peer_addr(tb, 1));
        }
      }
      mma_commit_pair(peer_addr(smem_u32(&drain_bar), 0));
      const uint64_t t0 = globaltimer();
      while (!mbar_test(smem_u32(&drain_bar), 0) && globaltimer() - t0 < kWaitLimitNs) {
      }
    }
  } else {
    // -------------------------------------------------- epilogue warps (both CTAs)
    const int quarter = warp & 3;  // TMEM lane quarter
    const int ep_tid = threadIdx.x - 64;
    const int col0 = ((warp - 2) >> 2) * kWarpCols;
    Epi e = epi;
    uint32_t i = 0;
    const uint32_t tempty_leader = peer_addr(smem_u32(&tempty_bar), 0);
    for (int64_t t = cid; t < num_tiles; t += ncl, ++i) {
      int64_t mt, nt;
      tile_mn(t, mt, nt);
      ColConst* cc = cols[i & 1];
      if (ep_tid < kTileN) e.column(nt * kTileN + ep_tid, cc[ep_tid]);
      const int64_t m = mt * kTileM + rank * 128 + quarter * 32 + lane;
      e.row(m);
      bounded_wait(smem_u32(&tfull_bar), i & 1, ctl, 14);
      // the epilogue warps leave together
      epi_bar(kEpiThreads);
      if (ep_tid == 0) epi_abort = abort_flag;
      epi_bar(kEpiThreads);
      if (epi_abort) break;
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col0;
      long long sum[kWarpCols];
#pragma unroll
      for (int c = 0; c < kWarpCols; c += 8) {
        int d[kDigits][8];
#pragma unroll
        for (int q = 0; q < kDigits; ++q) tmem_ld8(taddr + q * kTileN + c, d[q]);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          sum[c + k] = (long long)d[0][k] + (long long)d[1][k] * 256 + (long long)d[2][k] * 65536 +
                       (long long)d[3][k] * 16777216;
      }
      tc_fence_before();
      epi_bar(kEpiThreads);  // the whole accumulator of this CTA has been read
      if (ep_tid == 0) mbar_arrive_cluster(tempty_leader);
      const int64_t n0 = nt * kTileN + col0;
#pragma unroll
      for (int c = 0; c < kWarpCols; ++c) e.store(m, n0 + c, sum[c], cc[col0 + c]);
      e.stored(n0, lane);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the pair's MMAs or loads may touch it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kDigits * kTileN)
                 : "memory");
  }
}

template <class Epi>
cudaError_t run_i8(const CUtensorMap& tmA, const CUtensorMap& tmB, int64_t m, int64_t n, int64_t k,
                   const Epi& epi, TcStatus* status, int num_sms, cudaStream_t st) {
  const size_t dyn = (size_t)kStages * kStageBytes + 1024;
  auto kern = i8_pair_kernel<Epi>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  if (e != cudaSuccess) return e;
  const int64_t mt = (m + kTileM - 1) / kTileM, nt = (n + kTileN - 1) / kTileN;
  const int64_t tiles = mt * nt, pairs = num_sms / 2;
  if (tiles == 0 || pairs == 0) return cudaErrorInvalidValue;
  kern<<<2 * (unsigned)(tiles < pairs ? tiles : pairs), 64 + kEpiThreads, dyn, st>>>(
      tmA, tmB, mt, nt, (k + kStepK - 1) / kStepK, n, epi, status);
  return cudaGetLastError();
}

// ------------------------------------------------------------- operands --

// Balanced base-256 digits of q (|q| <= 127 (2^24 + 2^16 + 2^8 + 1)), lowest
// first, one byte each: with 128 added to the three low ones they are the
// bytes of a sum.
__device__ __forceinline__ uint32_t digits_of(int q) {
  return (uint32_t)(q + 0x00808080) ^ 0x00808080u;
}

// Rows of X [R][cols] (DIV: of X / phi of the column) as digit planes
// D [4][R][ld] and the row's unit 2^-k.  2^k puts the row's largest magnitude
// (rowmax, which may be a rounding below it) below 2^31 and the top digit within
// a byte.  A block takes 1024 columns of `rows` rows, a thread four neighbouring
// columns, so a reciprocal serves every row.  A row per block with a division
// and shifts for the bytes took 57 instructions an element and bound it (88% of
// the issue slots); the compress stage of 10,000 columns x 25,680 rows 3.73 ->
// 3.63 ms, the maximize stage of 12,800 x 25,680 2.92 -> 2.84 ms.
constexpr int kQuantRows = 8, kQuantStep = 4;

// 1 / d = r + rl, rl to first order in the rounding of r; x / d from them.
__device__ __forceinline__ void reciprocal(float d, float& r, float& rl) {
  r = 1.0f / d;
  rl = r * fmaf(-r, d, 1.0f);
}
__device__ __forceinline__ float quotient(float x, float r, float rl) { return fmaf(x, r, x * rl); }

template <bool DIV>
__global__ void __launch_bounds__(256) quant_rows_kernel(const float* X, const float* div,
                                                         const float* rowmax, int64_t R,
                                                         int64_t cols, int64_t ld, int rows,
                                                         int8_t* D, float* unit,
                                                         int32_t* flag, uint32_t* bits,
                                                         int32_t* count) {
  __shared__ float ups[kQuantRows];
  const int64_t chunks = (ld + 1023) / 1024, rb = blockIdx.x / chunks;
  const int64_t r0 = rb * rows, c0 = (blockIdx.x - rb * chunks) * 1024;
  if (threadIdx.x < rows && r0 + threadIdx.x < R) {
    const float mx = rowmax[r0 + threadIdx.x];
    const int ex = (int)((__float_as_uint(mx) >> 23) & 0xff) - 127;
    float up = 0.0f, one = 0.0f;  // a row of zeros (or denormals): all digits 0
    if (ex == 128) {
      one = __int_as_float(0x7fffffff);  // an infinite or NaN element: the row's sums are NaN
    } else if (ex > -127) {
      int k = 30 - ex;
      if (k > 126) k = 126;
      if (ldexpf(mx, k) > 2130706432.0f) --k;
      up = ldexpf(1.0f, k);
      one = ldexpf(1.0f, -k);
    }
    ups[threadIdx.x] = up;
    if (c0 == 0) unit[r0 + threadIdx.x] = one;
    if (c0 == 0 && flag) flag[r0 + threadIdx.x] = 0;
  }
  const int64_t j0 = c0 + 4 * threadIdx.x;
  float r[4], rl[4];
  if (DIV) {
#pragma unroll
    for (int i = 0; i < 4; ++i) reciprocal(j0 + i < cols ? div[j0 + i] : 1.0f, r[i], rl[i]);
  }
  __syncthreads();
  const uint32_t live = __ballot_sync(0xffffffffu, j0 < ld);
  if (j0 >= ld) return;
  const int64_t words = i8_bit_words(cols), word = 4 * (j0 / 128);
  const bool wide = cols % 4 == 0;  // then so is j0 < cols for the four columns
  for (int h = 0; h < rows; h += kQuantStep) {
    float v[kQuantStep][4];
#pragma unroll
    for (int k = 0; k < kQuantStep; ++k) {
      const float* x = X + (r0 + h + k) * cols + j0;
      const bool in = r0 + h + k < R;
      if (wide) {
        const float4 q = in && j0 < cols ? *reinterpret_cast<const float4*>(x)
                                         : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        v[k][0] = q.x, v[k][1] = q.y, v[k][2] = q.z, v[k][3] = q.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[k][i] = in && j0 + i < cols ? x[i] : 0.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < kQuantStep; ++k) {
      if (r0 + h + k >= R) break;
      const float up = ups[h + k];
      uint32_t w[4], rem[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float q = DIV ? quotient(v[k][i], r[i], rl[i]) : v[k][i];
        const float t = q * up;
        w[i] = digits_of(__float2int_rn(t));
        // 0 < t < 2^23: there may be a remainder
        if (DIV) rem[i] = __ballot_sync(live, __float_as_uint(t) - 1u < 0x4affffffu);
      }
      if (DIV && threadIdx.x % 32 == 0) {
        *reinterpret_cast<uint4*>(bits + (r0 + h + k) * words + word) =
            make_uint4(rem[0], rem[1], rem[2], rem[3]);
        const int n = __popc(rem[0]) + __popc(rem[1]) + __popc(rem[2]) + __popc(rem[3]);
        if (n) atomicAdd(count + r0 + h + k, n);
      }
      // four columns' digits to four digits' columns
      const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
      const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
      int8_t* o = D + (r0 + h + k) * ld + j0;
      const int64_t plane = R * ld;
      *reinterpret_cast<uint32_t*>(o) = __byte_perm(a, b, 0x5410);
      *reinterpret_cast<uint32_t*>(o + plane) = __byte_perm(a, b, 0x7632);
      *reinterpret_cast<uint32_t*>(o + 2 * plane) = __byte_perm(c, d, 0x5410);
      *reinterpret_cast<uint32_t*>(o + 3 * plane) = __byte_perm(c, d, 0x7632);
    }
  }
}

// U[r][j] += sum_p e_rp K_pj / T_r with e = P / phi - q unit, what launch_quant_rows
// left of an element (exact in FP32: q below 2^23 where there is a remainder, and
// all of the element where q is 0), for the rows that are flagged and inserted.
//
// A block takes a row at a time: the elements that may have a remainder are a bit
// each (launch_quant_rows), so it lists them, a thread an element; then a warp
// takes an element, or a part of one where there are few, and adds its pattern's
// photon list into the row's slice in shared memory.  With sharp posteriors few P
// are above zero: 2,000 x 25,680 at 128^2 (37% of the rows inserted, 53 remainders
// in the median one, 700 at most) 0.94 ms, the shared-memory additions, 3.4e11 a
// second; 10,000 x 25,680 at 64^2, poisson (34%, 3 and 284) 0.39 ms, latency; 64 x
// 420 at 16^2 14 us.  Without a flagged row a block reads its flags and ends: 2 us.
// Scanning the row of P for the elements: 1.2 to 1.4 ms; count bytes instead of
// photon lists: 2.9 ms at 128^2, every pixel of a pattern looked at.
constexpr int kSmallThreads = 512, kSmallWarps = kSmallThreads / 32;
constexpr int kSmallList = 384, kSmallUnroll = 4;
constexpr int64_t kSmallPixels = 48 << 10;  // of a slice in shared memory

// Blocks that share a row of `count` elements: with broad posteriors a row may have
// a thousand (1,000 x 3,240 at 32^2 gaussian: one block took 95 us over it).
constexpr int kSmallParts = 8, kSmallShare = 128;
__device__ __forceinline__ int small_parts(int count) {
  const int n = count / kSmallShare;
  return n < 1 ? 1 : n < kSmallParts ? n : kSmallParts;
}

__global__ void __launch_bounds__(kSmallThreads, 3) small_terms_kernel(const I8SmallArgs a,
                                                              const int64_t tile) {
  extern __shared__ float slice[];  // [tile]
  __shared__ uint32_t need[kSmallWarps];
  __shared__ int part[kSmallWarps];
  __shared__ int32_t lp[kSmallList], ln[kSmallList];
  __shared__ float le[kSmallList];
  __shared__ int64_t lb[kSmallList];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t words = i8_bit_words(a.N);
  const int64_t units = a.R * kSmallParts;
  for (int64_t base = blockIdx.x; base < units; base += (int64_t)gridDim.x * kSmallThreads) {
    const int64_t mine = base + (int64_t)threadIdx.x * gridDim.x, row = mine % a.R;
    bool n = false;
    if (mine < units) {
      const float T = a.T[row];
      n = a.flag[row] != 0 && (a.Tskip ? a.Tskip[row] : T) > 1e-10f && T > 0.0f &&
          mine / a.R < small_parts(a.count[row]);
    }
    const uint32_t b = __ballot_sync(0xffffffffu, n);
    if (lane == 0) need[w] = b;
    if (!__syncthreads_or(n)) continue;
    // (row, part, pixel tile) after another, the same for every thread
    for (int i = 0; i < kSmallWarps; ++i)
      for (uint32_t rest = need[i]; rest; rest &= rest - 1)
        for (int64_t j0 = 0; j0 < a.npa; j0 += tile) {
          const int64_t unit = base + (32 * i + __ffs(rest) - 1) * (int64_t)gridDim.x;
          const int64_t r = unit % a.R, share = unit / a.R;
          // elements lo .. hi - 1 of the row's, `seen` of them before these words
          const int count = a.count[r], shares = small_parts(count);
          const int lo = (int)(count * share / shares), hi = (int)(count * (share + 1) / shares);
          int seen = 0;
          const int px = (int)(a.npa - j0 < tile ? a.npa - j0 : tile);
          const float one = a.unit[r], up = one > 0.0f ? 1.0f / one : 0.0f;
          bool any = false;
          for (int64_t g0 = 0; g0 < words; g0 += kSmallThreads) {
            const int64_t g = g0 + threadIdx.x;
            const uint32_t word = g < words ? a.bits[r * words + g] : 0u;
            // each thread's place among the elements of these words
            int place = __popc(word), total = 0;
            const int own = place;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int v = __shfl_up_sync(0xffffffffu, place, o);
              if (lane >= o) place += v;
            }
            if (lane == 31) part[w] = place;
            __syncthreads();
            place -= own;
            for (int k = 0; k < kSmallWarps; ++k) {
              const int v = part[k];
              if (k < w) place += v;
              total += v;
            }
            const int from = lo > seen ? lo - seen : 0, to = hi - seen < total ? hi - seen : total;
            if (from < to && !any) {
              for (int j = threadIdx.x; j < px; j += kSmallThreads) slice[j] = 0.0f;
              any = true;
            }
            for (int done = from; done < to; done += kSmallList) {
              const int m = to - done < kSmallList ? to - done : kSmallList;
              int at = place - done;
              for (uint32_t z = word; z; z &= z - 1, ++at)
                if ((unsigned)at < (unsigned)m)
                  lp[at] = (int32_t)((g >> 2) * 128 + 4 * (__ffs(z) - 1) + (g & 3));
              __syncthreads();
              for (int q = threadIdx.x; q < m; q += kSmallThreads) {
                const int64_t p = lp[q], beg = a.kbeg[p];
                float rc, rl;
                reciprocal(a.phi[p], rc, rl);
                const float x = quotient(a.P[r * a.N + p], rc, rl);
                le[q] = fmaf(-(float)__float2int_rn(x * up), one, x);
                lb[q] = beg;
                ln[q] = (int)(a.kend[p] - beg);
              }
              __syncthreads();
              // few elements: several warps each, a part of its list
              const int parts = m < kSmallWarps ? kSmallWarps / m : 1;
              for (int u = w; u < m * parts; u += kSmallWarps) {
                const int q = u % m, nq = ln[q];
                const int64_t t0 = lb[q];
                const float x = le[q];
                const int step = 32 * kSmallUnroll;
                for (int t = u / m * step + lane; t < nq; t += parts * step) {
                  int j[kSmallUnroll];
                  float c[kSmallUnroll];
#pragma unroll
                  for (int z = 0; z < kSmallUnroll; ++z) {
                    const bool in = t + 32 * z < nq;
                    j[z] = in ? a.kidx[t0 + t + 32 * z] - (int)j0 : -1;
                    c[z] = in ? a.kval[t0 + t + 32 * z] : 0.0f;
                  }
#pragma unroll
                  for (int z = 0; z < kSmallUnroll; ++z)
                    if ((unsigned)j[z] < (unsigned)px) atomicAdd(slice + j[z], x * c[z]);
                }
              }
              __syncthreads();  // lists and `part` are written again
            }
            if (from >= to) __syncthreads();
            seen += total;
          }
          if (!any) continue;
          const float T = a.T[r], inv = T > 1e-30f ? 1.0f / T : 1.0f;
          float* o = a.U + r * a.npa + j0;
          for (int j = threadIdx.x; j < px; j += kSmallThreads * kSmallUnroll) {
            float u[kSmallUnroll];
#pragma unroll
            for (int z = 0; z < kSmallUnroll; ++z)
              u[z] = j + z * kSmallThreads < px ? o[j + z * kSmallThreads] : 0.0f;
#pragma unroll
            for (int z = 0; z < kSmallUnroll; ++z)
              if (j + z * kSmallThreads < px) {
                const float x = slice[j + z * kSmallThreads];
                if (shares == 1)
                  o[j + z * kSmallThreads] = fmaf(x, inv, u[z]);
                else if (x != 0.0f)
                  atomicAdd(o + j + z * kSmallThreads, x * inv);
              }
          }
          __syncthreads();
        }
    __syncthreads();  // `need` is written again
  }
}

// rowmax[r] = the largest |X| (or |X / div|, within a rounding, as
// quant_rows_kernel allows) of row r; a NaN stays the largest.  One block per row.
__global__ void __launch_bounds__(256) row_maxima_kernel(const float* X, const float* div,
                                                         int64_t cols, float* rowmax) {
  __shared__ uint32_t red[8];
  const float* x = X + blockIdx.x * cols;
  uint32_t mx = 0;
  for (int64_t j = threadIdx.x; j < cols; j += 256) {
    const float v = div ? x[j] * (1.0f / div[j]) : x[j];
    mx = max(mx, __float_as_uint(fabsf(v)));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) mx = max(mx, red[k]);
    rowmax[blockIdx.x] = __uint_as_float(mx);
  }
}

// Counts K [N][npa] as bytes by pattern (K8 [planes][N][ldK]) and by pixel
// (Kt8 [planes][npa][ldT]), base-128 digits when planes == 2, and each pixel's
// total (kI8MaxTotal keeps it below 2^32).
__global__ void pack_counts_i8_kernel(const float* K, int64_t N, int64_t npa, int planes,
                                      int64_t ldK, int64_t ldT, int8_t* K8, int8_t* Kt8,
                                      uint32_t* ktot) {
  __shared__ int tile[32][33];
  const int64_t jb = (npa + 31) / 32;
  const int64_t j0 = blockIdx.x % jb * 32, p0 = blockIdx.x / jb * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int i = ty; i < 32; i += 8) {
    const int64_t p = p0 + i, j = j0 + tx;
    const int k = (p < N && j < npa) ? (int)K[p * npa + j] : 0;
    tile[i][tx] = k;
    if (p < N && j < npa)
      for (int s = 0; s < planes; ++s)
        K8[((int64_t)s * N + p) * ldK + j] = (int8_t)((k >> (7 * s)) & 127);
  }
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int64_t j = j0 + i, p = p0 + tx;
    const uint32_t sum = __reduce_add_sync(0xffffffffu, (uint32_t)tile[tx][i]);
    if (tx == 0 && j < npa && sum) atomicAdd(ktot + j, sum);
    if (p < N && j < npa)
      for (int s = 0; s < planes; ++s)
        Kt8[((int64_t)s * npa + j) * ldT + p] = (int8_t)((tile[tx][i] >> (7 * s)) & 127);
  }
}

// The photon lists of the patterns: pattern p's non-zero pixels and counts at
// beg[p] .. end[p] - 1, the lists one after the other in no particular order of
// patterns (total[0]: 0 on entry), so no scan over them is needed.  One warp per
// pattern, which counts and then fills.
__global__ void photon_lists_kernel(const float* K, int64_t N, int64_t npa, int64_t* beg,
                                    int64_t* end, int32_t* idx, float* val,
                                    unsigned long long* total) {
  const int64_t p = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (p >= N) return;
  const float* row = K + p * npa;
  uint32_t n = 0;
  for (int64_t j = lane; j < npa; j += 32) n += row[j] != 0.0f;
  n = __reduce_add_sync(0xffffffffu, n);
  unsigned long long at = 0;
  if (lane == 0) {
    at = atomicAdd(total, (unsigned long long)n);
    beg[p] = (int64_t)at;
    end[p] = (int64_t)at + n;
  }
  at = __shfl_sync(0xffffffffu, at, 0);
  for (int64_t j0 = 0; j0 < npa; j0 += 32) {
    const int64_t j = j0 + lane;
    const float k = j < npa ? row[j] : 0.0f;
    const uint32_t nz = __ballot_sync(0xffffffffu, k != 0.0f);
    if (k != 0.0f) {
      const unsigned long long o = at + __popc(nz & ((1u << lane) - 1u));
      idx[o] = (int32_t)j;
      val[o] = k;
    }
    at += __popc(nz);
  }
}

// out[0] = bits of the largest entry, out[1] += entries that are not integers
// in [0, limit], out[2] += entries that are negative, NaN or infinite; nonzero[0]
// += the entries that are not 0.
__global__ void count_range_kernel(const float* x, int64_t n, float limit, unsigned int* out,
                                   unsigned long long* nonzero) {
  unsigned int mx = 0, odd = 0, bad = 0, nz = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float v = x[i];
    if (!(v >= 0.0f && v <= FLT_MAX)) {
      ++bad;
      continue;
    }
    if (!(v <= limit && v == floorf(v))) ++odd;
    if (v != 0.0f) ++nz;
    mx = max(mx, __float_as_uint(fabsf(v)));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  odd = __reduce_add_sync(0xffffffffu, odd);
  bad = __reduce_add_sync(0xffffffffu, bad);
  nz = __reduce_add_sync(0xffffffffu, nz);  // fewer than 2^32 a warp
  if ((threadIdx.x & 31) == 0) {
    if (mx) atomicMax(out, mx);
    if (odd) atomicAdd(out + 1, odd);
    if (bad) atomicAdd(out + 2, bad);
    if (nz) atomicAdd(nonzero, (unsigned long long)nz);
  }
}

}  // namespace

bool i8_encode(CUtensorMap* tm, const void* base, int64_t inner, int64_t rows, int64_t ld,
               bool counts) {
  return tc_encode_2d_bytes(tm, base, (uint64_t)inner, (uint64_t)rows, (uint64_t)ld,
                            counts ? 128 : kTileN / 2, kStepK);
}

cudaError_t launch_i8_loglik(const CUtensorMap& tmK, const CUtensorMap& tmX, int64_t npa,
                             const I8LLArgs& a, TcStatus* status, int num_sms, cudaStream_t st) {
  EpiLL e;
  e.a = a;
  return run_i8(tmK, tmX, a.N, a.R, npa, e, status, num_sms, st);
}

cudaError_t launch_i8_slices(const CUtensorMap& tmKt, const CUtensorMap& tmX, int64_t N,
                             const I8UArgs& a, TcStatus* status, int num_sms, cudaStream_t st) {
  EpiU e;
  e.a = a;
  return run_i8(tmKt, tmX, a.npa, a.R, N, e, status, num_sms, st);
}

cudaError_t launch_quant_rows(const float* X, const float* div, const float* rowmax, int64_t R,
                              int64_t cols, int64_t ld, int8_t* D, float* unit, int32_t* flag,
                              uint32_t* bits, int32_t* count, cudaStream_t st) {
  if (R <= 0) return cudaSuccess;
  if (ld % 16 != 0 || ld < cols || (div && !(flag && bits && count))) return cudaErrorInvalidValue;
  int rows = kQuantRows;
  const int64_t chunks = (ld + 1023) / 1024;
  while (rows > kQuantStep && chunks * ((R + rows - 1) / rows) < 4 * 148) rows /= 2;
  const unsigned grid = (unsigned)(chunks * ((R + rows - 1) / rows));
  if (div)
    quant_rows_kernel<true><<<grid, 256, 0, st>>>(X, div, rowmax, R, cols, ld, rows, D, unit,
                                                    flag, bits, count);
  else
    quant_rows_kernel<false><<<grid, 256, 0, st>>>(X, div, rowmax, R, cols, ld, rows, D, unit,
                                                    flag, bits, count);
  return cudaGetLastError();
}

cudaError_t launch_small_terms(const I8SmallArgs& a, int num_sms, cudaStream_t st) {
  if (a.R <= 0 || a.N <= 0) return cudaSuccess;
  const int64_t tile = std::min<int64_t>((a.npa + 31) / 32 * 32, kSmallPixels);
  const size_t smem = sizeof(float) * (size_t)tile;
  const cudaError_t e = cudaFuncSetAttribute(
      small_terms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // as many blocks an SM, up to three, as slices and lists (20 bytes an element) fit
  const int64_t per_sm = std::clamp<int64_t>((227 << 10) / (smem + 20 * kSmallList + 1400), 1, 3);
  const int64_t grid = std::min<int64_t>(a.R * kSmallParts, per_sm * num_sms);
  small_terms_kernel<<<(unsigned)grid, kSmallThreads, smem, st>>>(a, tile);
  return cudaGetLastError();
}

cudaError_t launch_row_maxima(const float* X, const float* div, int64_t R, int64_t cols,
                              float* rowmax, cudaStream_t st) {
  if (R <= 0) return cudaSuccess;
  row_maxima_kernel<<<(unsigned)R, 256, 0, st>>>(X, div, cols, rowmax);
  return cudaGetLastError();
}

cudaError_t launch_pack_counts_i8(const float* K, int64_t N, int64_t npa, int planes, int64_t ldK,
                                  int64_t ldT, int8_t* K8, int8_t* Kt8, uint32_t* ktot,
                                  cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(ktot, 0, sizeof(uint32_t) * npa, st);
  if (e != cudaSuccess) return e;
  const int64_t grid = ((npa + 31) / 32) * ((N + 31) / 32);
  pack_counts_i8_kernel<<<(unsigned)grid, dim3(32, 8), 0, st>>>(K, N, npa, planes, ldK, ldT, K8,
                                                               Kt8, ktot);
  return cudaGetLastError();
}

cudaError_t launch_photon_lists(const float* K, int64_t N, int64_t npa, int64_t* beg, int64_t* end,
                                int32_t* idx, float* val, unsigned long long* total,
                                cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(total, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess || N <= 0) return e;
  photon_lists_kernel<<<(unsigned)((N + 7) / 8), 256, 0, st>>>(K, N, npa, beg, end, idx, val,
                                                               total);
  return cudaGetLastError();
}

cudaError_t launch_count_range(const float* x, int64_t n, float limit, CountRange* out,
                               cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(out, 0, sizeof(CountRange), st);
  if (e != cudaSuccess || n <= 0) return e;
  count_range_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 1184), 256, 0, st>>>(
      x, n, limit, &out->largest, &out->nonzero);
  return cudaGetLastError();
}

}  // namespace emc
