// The MATLAB v5 uniform stream on the GPU (v5_uniform.cuh states the algorithm).
#include "v5_uniform.cuh"

#include <algorithm>
#include <mutex>

namespace ps2 {
namespace {

constexpr uint32_t kSeed = 2005;
constexpr int kKeptRows = 320;  // table rows kept by the process: 84 million draws

__host__ __device__ inline uint32_t xs32(uint32_t v) {
  v ^= v << 13;
  v ^= v >> 17;
  v ^= v << 5;
  return v;
}

V5Num v5_pow(V5Num base, int64_t e) {
  V5Num r{};
  r.d[0] = 1;
  for (; e > 0; e >>= 1) {
    if (e & 1) r = v5_mulmod(r, base);
    base = v5_mulmod(base, base);
  }
  return r;
}

// b mod m, and a = b^-1 mod m: a is what one draw multiplies Y by, so it is
// the state after one draw from Y = 1
V5Num v5_one() {
  V5Num r{};
  r.d[0] = 1;
  return r;
}
V5Num v5_a() {
  V5Num y = v5_one();
  v5_emit(y);
  return y;
}

// Y of the seeded generator: its 32 words, the last 27 of them in use
V5Num v5_seeded() {
  uint64_t w[32];
  uint32_t s = kSeed;
  for (int k = 0; k < 32; ++k) {
    uint64_t x = 0;
    for (int b = 0; b < 53; ++b) {
      s = xs32(s);
      x = (x << 1) | ((s >> 19) & 1u);
    }
    w[k] = x;
  }
  const uint64_t* x = w + 5;
  V5Num y;
  int64_t c = 0;
  for (int i = 0; i < kV5Long; ++i) {
    int64_t v = c + static_cast<int64_t>(x[i]);
    if (i < kV5Short) v -= static_cast<int64_t>(x[i + kV5Long - kV5Short]);
    y.d[i] = static_cast<uint64_t>(v) & kV5Mask;
    c = v >> 53;
  }
  if (c < 0) {  // below zero: + m
    c = 0;
    for (int i = 0; i < kV5Long; ++i) {
      int64_t v = c + static_cast<int64_t>(y.d[i]) + (i == 0 ? 1 : 0) +
                  (i >= kV5Short ? static_cast<int64_t>(kV5Mask) : 0);
      y.d[i] = static_cast<uint64_t>(v) & kV5Mask;
      c = v >> 53;
    }
  }
  return y;
}

V5Tables g_tables;
V5Num g_row_step;
std::once_flag g_once;

void make_tables() {
  const V5Num a = v5_a();
  const V5Num seg = v5_pow(a, kV5Segment);
  g_tables.step.assign(1, v5_one());
  for (int r = 1; r < kV5Row; ++r) g_tables.step.push_back(v5_mulmod(g_tables.step.back(), seg));
  g_row_step = v5_mulmod(g_tables.step.back(), seg);
  // 27 draws back: times b^27
  V5Num b{};
  b.d[1] = 1;
  g_tables.start.assign(1, v5_mulmod(v5_seeded(), v5_pow(b, kV5Long)));
  while (static_cast<int>(g_tables.start.size()) < kKeptRows)
    g_tables.start.push_back(v5_mulmod(g_tables.start.back(), g_row_step));
  uint32_t m[32];
  for (int k = 0; k < 32; ++k) m[k] = xs32(1u << k);
  auto apply = [](const uint32_t* col, uint32_t v) {
    uint32_t r = 0;
    for (int k = 0; k < 32; ++k)
      if ((v >> k) & 1u) r ^= col[k];
    return r;
  };
  for (int e = 1; e < kV5Segment; e *= 2) {
    uint32_t q[32];
    for (int k = 0; k < 32; ++k) q[k] = apply(m, m[k]);
    std::copy(q, q + 32, m);
  }
  for (int i = 0; i < 32; ++i) {
    g_tables.jump.insert(g_tables.jump.end(), m, m + 32);
    uint32_t q[32];
    for (int k = 0; k < 32; ++k) q[k] = apply(m, m[k]);
    std::copy(q, q + 32, m);
  }
}

// One thread per segment. What bounds it is a thread's own chain (the borrow of
// a draw enters the next one) and the segment's start. 18 million draws (300,000
// rows x 60) take 0.096 ms; one host thread took about 190 ms, and 13 ms more went
// into the upload of the matrix.
__global__ void __launch_bounds__(64) k_v5_uniform(const V5Num* __restrict__ step, const V5Num* __restrict__ start,
                                                   const uint32_t* __restrict__ jump, double scale,
                                                   double* __restrict__ out, int64_t n) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t n0 = t * kV5Segment;
  if (n0 >= n) return;
  uint64_t x[32];  // word n sits in slot n mod 32, as in the reference's ring
  int64_t borrow;
  {
    V5Num y = v5_mulmod(start[t / kV5Row], step[t % kV5Row]);
    uint64_t w[kV5Long];
    for (int i = 0; i < kV5Long; ++i) w[i] = v5_emit(y);
    borrow = static_cast<int64_t>((y.d[0] - w[0] + w[kV5Long - kV5Short]) & kV5Mask);
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = i < 5 ? 0 : w[i - 5];
  }
  uint32_t j = kSeed;
  for (int i = 0; i < 32 && (t >> i) != 0; ++i) {
    if (((t >> i) & 1) == 0) continue;
    uint32_t r = 0;
    for (int k = 0; k < 32; ++k) r ^= ((j >> k) & 1u) ? jump[32 * i + k] : 0u;
    j = r;
  }
  const int64_t left = n - n0 < kV5Segment ? n - n0 : kV5Segment;
  for (int64_t i0 = 0; i0 < left; i0 += 32) {
    double even = 0.0;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int64_t v = static_cast<int64_t>(x[(i + 20) & 31]) - static_cast<int64_t>(x[(i + 5) & 31]) - borrow;
      borrow = v < 0 ? 1 : 0;
      x[i] = static_cast<uint64_t>(v) & kV5Mask;
      // the mantissa bits exchanged with two xorshift words (a zero word gives
      // the mask itself, times 2^-53)
      const uint32_t lo = j;
      j = xs32(j);
      const uint64_t mask = ((static_cast<uint64_t>(j) << 32) & (kV5Mask >> 1)) ^ lo;
      const double u = static_cast<double>(x[i]) * 1.1102230246251565e-16;
      const double z = x[i] != 0 ? __longlong_as_double(__double_as_longlong(u) ^ static_cast<long long>(mask))
                                 : static_cast<double>(mask) * 1.1102230246251565e-16;
      const double f = __dmul_rn(z, scale);
      const int64_t at = i0 + i;
      if (i & 1) {
        if (at < left)
          *reinterpret_cast<double2*>(out + n0 + at - 1) = make_double2(even, f);
        else if (at - 1 < left)
          out[n0 + at - 1] = even;
      } else {
        even = f;
      }
    }
  }
}

}  // namespace

void v5_tables(int64_t n, V5Tables* out) {
  std::call_once(g_once, make_tables);
  const int64_t per_row = static_cast<int64_t>(kV5Segment) * kV5Row;
  const int64_t rows = std::max<int64_t>((n + per_row - 1) / per_row, 1);
  out->step = g_tables.step;
  out->jump = g_tables.jump;
  out->start.assign(g_tables.start.begin(),
                    g_tables.start.begin() + static_cast<size_t>(std::min<int64_t>(rows, kKeptRows)));
  while (static_cast<int64_t>(out->start.size()) < rows)
    out->start.push_back(v5_mulmod(out->start.back(), g_row_step));
}

cudaError_t launch_v5_uniform(const V5Num* step, const V5Num* start, const uint32_t* jump, double scale, double* out,
                              int64_t n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t threads = (n + kV5Segment - 1) / kV5Segment;
  k_v5_uniform<<<static_cast<unsigned>((threads + 63) / 64), 64, 0, st>>>(step, start, jump, scale, out, n);
  return cudaGetLastError();
}

}  // namespace ps2
