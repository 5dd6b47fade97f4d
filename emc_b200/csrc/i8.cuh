// FP32 contexts' contractions on the byte tensor cores (kernels_i8.cu): launch
// interface.  X is quantised row by row into four digit planes D [4][R][ld]
// (launch_quant_rows); the counts are bytes, in two base-128 planes when one
// exceeds 127 (the contraction then runs twice, I8_HIGH then I8_LOW).
#pragma once
#include <cstdint>

#include "tc.cuh"

namespace emc {

constexpr int kI8Digits = 4;
constexpr int kI8MaxCount = 127;            // one plane
constexpr int kI8MaxCount2 = 127 * 128 + 127;  // two
// Elements of a row of X per unit of count: 32-bit sums hold 128 x the total
// count of a row of the count operand.
constexpr double kI8MaxTotal = 2147483647.0 / 128.0;

enum I8Pass { I8_ONLY = 0, I8_HIGH = 1, I8_LOW = 2 };

struct I8LLArgs {
  int64_t R, N;
  int poisson, pass;
  double mult;             // 1, or 128 (I8_HIGH)
  const float* unit;       // [R]
  const float* scaling;    // [N]
  const double* rowstat;   // [R] sum W or sum S^2
  const double* patstat;   // [N] gaussian: sum K^2
  double gauss_inv;
  double* LL;              // [R][N]
};
struct I8UArgs {
  int64_t R, npa;
  int pass;
  double mult;
  const float* unit;       // [R]
  const float* T;          // [R]
  float* U;                // [R][npa]
  const uint32_t* ktot;    // [npa] photons at the pixel over all patterns
  int32_t* flag;           // [R] set where a pixel's sum has few digits (launch_small_terms)
};
// What the fixed point of a row leaves out of its slice sums: the remainders of
// P / phi (all of it below half a unit), added to U in the rows that are flagged
// and inserted (Tskip or T above 1e-10).
struct I8SmallArgs {
  int64_t R, N, npa;
  const float* P;          // [R][N]
  const float* phi;        // [N]
  const float* unit;       // [R]
  const float *T, *Tskip;  // [R]
  const int32_t* flag;     // [R]
  const uint32_t* bits;    // of launch_quant_rows,
  const int32_t* count;    // with their number [R]
  const int64_t *kbeg, *kend;  // photon lists: pattern p's are kbeg[p] .. kend[p] - 1
  const int32_t* kidx;
  const float* kval;
  float* U;                // [R][npa]
};

// Tensor map of a byte operand: the counts (inner = contraction extent) or
// the digit planes (rows = 4 R).  ld is a multiple of 16 bytes; bytes between
// inner and ld are never read.
bool i8_encode(CUtensorMap* tm, const void* base, int64_t inner, int64_t rows, int64_t ld,
               bool counts);
cudaError_t launch_i8_loglik(const CUtensorMap& tmK, const CUtensorMap& tmX, int64_t npa,
                             const I8LLArgs& a, TcStatus* status, int num_sms, cudaStream_t st);
cudaError_t launch_i8_slices(const CUtensorMap& tmKt, const CUtensorMap& tmX, int64_t N,
                             const I8UArgs& a, TcStatus* status, int num_sms, cudaStream_t st);
cudaError_t launch_small_terms(const I8SmallArgs& a, int num_sms, cudaStream_t st);
// rowmax [R]: the largest |X| of the row (after the division by div[column]).
// With div also: flag [R] zeroed, count [R] (zeros on entry) the number of, and bits [R][i8_bit_words(cols)], 16-byte
// aligned: bit l of word 4 g + i is set where element 128 g + 4 l + i of the row
// may have a remainder.
inline __host__ __device__ int64_t i8_bit_words(int64_t cols) { return 4 * ((cols + 127) / 128); }
cudaError_t launch_quant_rows(const float* X, const float* div, const float* rowmax, int64_t R,
                              int64_t cols, int64_t ld, int8_t* D, float* unit, int32_t* flag,
                              uint32_t* bits, int32_t* count, cudaStream_t st);
// The same rowmax from X and div.
cudaError_t launch_row_maxima(const float* X, const float* div, int64_t R, int64_t cols,
                              float* rowmax, cudaStream_t st);
cudaError_t launch_pack_counts_i8(const float* K, int64_t N, int64_t npa, int planes, int64_t ldK,
                                  int64_t ldT, int8_t* K8, int8_t* Kt8, uint32_t* ktot,
                                  cudaStream_t st);
// Photon lists of counts K [N][npa] (as I8SmallArgs); total: one word of scratch.
cudaError_t launch_photon_lists(const float* K, int64_t N, int64_t npa, int64_t* beg, int64_t* end,
                                int32_t* idx, float* val, unsigned long long* total,
                                cudaStream_t st);
struct CountRange {
  unsigned int largest;  // its bits
  unsigned int odd;      // entries that are not integers in [0, limit]
  unsigned int bad;      // entries that are negative, NaN or infinite
  unsigned int pad;
  unsigned long long nonzero;
};
cudaError_t launch_count_range(const float* x, int64_t n, float limit, CountRange* out,
                               cudaStream_t st);

}  // namespace emc
