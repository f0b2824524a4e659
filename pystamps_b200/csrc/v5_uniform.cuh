// MATLAB rand('state', seed) / v5 uniform generator (native_stage2.rs:1785-1873)
// as many independent segments of one stream, so that the GPU can draw it.
//
// The generator is a subtract-with-borrow recurrence on 53-bit words,
//   x_n = x_{n-12} - x_{n-27} - c  (mod b = 2^53, c the borrow),
// whose word then has its mantissa bits exchanged with a xorshift-32 sequence
// that advances once a draw. Subtract-with-borrow is a multiplicative
// congruential sequence in disguise (Marsaglia and Zaman, "A new class of random
// number generators", Ann. Appl. Probab. 1, 1991; Tezuka, L'Ecuyer and Couture,
// ACM TOMACS 3, 1993): with x_0 the oldest of the last 27 words,
//   Y = sum_{k<27} x_k b^k - sum_{k<12} x_{k+15} b^k + c,   m = b^27 - b^12 + 1,
// a draw is Y <- Y b^-1 mod m, and it emits the digit d = -Y mod b because
// Y + d m is then divisible by b. A segment that starts at draw n therefore
// takes Y a^(n - 27) (a = b^-1 mod m), emits the 27 words before its start and
// goes on with the plain recurrence. xorshift-32 is linear over GF(2), so its
// state jumps by 32 x 32 bit matrices.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace ps2 {

constexpr int kV5Long = 27, kV5Short = 12;
constexpr uint64_t kV5Mask = (uint64_t(1) << 53) - 1;
// Draws per segment (a thread's share) and segments per table row. 1,024 draws
// against the start of a segment (one product mod m and 27 digits, about 15,000
// instructions): a 300,000 x 60 matrix gives 17,600 threads.
constexpr int kV5Segment = 1024;
constexpr int kV5Row = 256;

struct V5Num {
  uint64_t d[kV5Long];  // base-2^53 digits, least significant first, below m
};

// a b mod m. b^27 = b^12 - 1 (mod m): the upper 27 digits of the product fold
// onto the lower ones, twice; then at most one subtraction of m is left.
__host__ __device__ inline V5Num v5_mulmod(const V5Num& a, const V5Num& b) {
  uint64_t p[2 * kV5Long];
  unsigned __int128 acc = 0;
  for (int k = 0; k < 2 * kV5Long - 1; ++k) {
    const int lo = k < kV5Long ? 0 : k - kV5Long + 1, hi = k < kV5Long ? k : kV5Long - 1;
    for (int i = lo; i <= hi; ++i) acc += static_cast<unsigned __int128>(a.d[i]) * b.d[k - i];
    p[k] = static_cast<uint64_t>(acc) & kV5Mask;
    acc >>= 53;
  }
  p[2 * kV5Long - 1] = static_cast<uint64_t>(acc);
  // first fold: digits 27 + k (k < 27) go to 12 + k and, negated, to k
  constexpr int kTop = kV5Long + kV5Short;  // 39 digits hold the folded value
  uint64_t t[kTop];
  int64_t c = 0;
  for (int i = 0; i < kTop; ++i) {
    int64_t v = c;
    if (i < kV5Long) v += static_cast<int64_t>(p[i]) - static_cast<int64_t>(p[kV5Long + i]);
    if (i >= kV5Short) v += static_cast<int64_t>(p[kV5Long + i - kV5Short]);
    t[i] = static_cast<uint64_t>(v) & kV5Mask;
    c = v >> 53;
  }
  // second fold: the 12 digits above the 27th
  V5Num r;
  c = 0;
  for (int i = 0; i < kV5Long; ++i) {
    int64_t v = c + static_cast<int64_t>(t[i]);
    if (i < kV5Short) v -= static_cast<int64_t>(t[kV5Long + i]);
    if (i >= kV5Short && i < 2 * kV5Short) v += static_cast<int64_t>(t[kV5Long + i - kV5Short]);
    r.d[i] = static_cast<uint64_t>(v) & kV5Mask;
    c = v >> 53;
  }
  // a carry of b^27 = b^12 - 1, or a value in [m, b^27): both subtract m once
  // (m's digits are 1, 0 x 11, (b - 1) x 15)
  bool over = c != 0;
  if (!over) {
    over = true;
    for (int i = kV5Short; i < kV5Long; ++i) over = over && r.d[i] == kV5Mask;
    if (over) {
      bool low = r.d[0] >= 1;
      for (int i = 1; i < kV5Short; ++i) low = low || r.d[i] != 0;
      over = low;
    }
  }
  if (over) {
    c = 0;
    for (int i = 0; i < kV5Long; ++i) {
      int64_t v = c + static_cast<int64_t>(r.d[i]);
      if (i == 0) v -= 1;
      if (i >= kV5Short) v -= static_cast<int64_t>(kV5Mask);
      r.d[i] = static_cast<uint64_t>(v) & kV5Mask;
      c = v >> 53;
    }
  }
  return r;
}

// One draw of Y: its digit, and Y <- (Y + d m) / b, digit by digit.
__host__ __device__ inline uint64_t v5_emit(V5Num& y) {
  const uint64_t d = (0 - y.d[0]) & kV5Mask;
  int64_t c = y.d[0] != 0 ? 1 : 0;  // y_0 + d is 0 or b
  for (int i = 1; i < kV5Long; ++i) {
    int64_t v = c + static_cast<int64_t>(y.d[i]);
    if (i == kV5Short) v -= static_cast<int64_t>(d);
    y.d[i - 1] = static_cast<uint64_t>(v) & kV5Mask;
    c = v >> 53;
  }
  y.d[kV5Long - 1] = static_cast<uint64_t>(c + static_cast<int64_t>(d));
  return d;
}

// Start of segment t = kV5Row q + r: start[q] step[r] (mod m), and the
// xorshift state jump[0..31]^(bits of t) applied to the seed.
struct V5Tables {
  std::vector<V5Num> step;       // [kV5Row] a^(kV5Segment r)
  std::vector<V5Num> start;      // [rows] Y a^(kV5Segment kV5Row q - 27)
  std::vector<uint32_t> jump;    // [32][32] columns of the xorshift matrix to the power kV5Segment 2^i
};
// The tables of seed 2005 for a stream of n draws.
void v5_tables(int64_t n, V5Tables* out);
// out[i] = scale * draw i of seed 2005, i < n; the tables of v5_tables in device memory
cudaError_t launch_v5_uniform(const V5Num* step, const V5Num* start, const uint32_t* jump, double scale, double* out,
                              int64_t n, cudaStream_t st);

}  // namespace ps2
