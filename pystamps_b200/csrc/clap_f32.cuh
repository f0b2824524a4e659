// CLAP window arithmetic in FP32, one warp per window and interferogram.
//
// The window kernels are bound by instruction issue and by instruction fetch: the
// straight-line code of four unrolled transforms, smoothing and median is streamed
// through once per window, so both the instructions executed and those stored
// count. One transform body serves all four passes: a lane always transforms its
// own row of the tile, a pass that goes on along the other axis stores its result
// transposed, and the inverse passes run the forward body on data whose real and
// imaginary parts are exchanged. Stages 1 to 4 of the 32 points work on packed
// FP32x2 values (points 2 m and 2 m + 1, whose butterflies and factors are the same
// there), one instruction for two. Every operation and its rounding is that of the
// plain radix-2 passes (fft_pass_t), with the quarter turn taken as exactly -i (its
// rounded cosine, 6e-17, is below the rounding of any sum it would enter).
#pragma once

#include "phase_math.cuh"
#include "ps2_device.cuh"
#include "ps2_kernels.cuh"

namespace ps2 {

__device__ __forceinline__ float2 sub2(const float2 a, const float2 b) {
  float2 r;
  asm("{.reg .b64 a, b, c; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; sub.rn.f32x2 c, a, b; mov.b64 {%0, %1}, c;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// cos(2 pi k / 32) and sin(2 pi k / 32), k < 16
static __constant__ float kCos32[16] = {
    0x1.0000000000000p+0f, 0x1.f6297c0000000p-1f, 0x1.d906bc0000000p-1f, 0x1.a9b6620000000p-1f,
    0x1.6a09e60000000p-1f, 0x1.1c73b40000000p-1f, 0x1.87de2a0000000p-2f, 0x1.8f8b840000000p-3f,
    0.f, -0x1.8f8b840000000p-3f, -0x1.87de2a0000000p-2f, -0x1.1c73b40000000p-1f,
    -0x1.6a09e60000000p-1f, -0x1.a9b6620000000p-1f, -0x1.d906bc0000000p-1f, -0x1.f6297c0000000p-1f};
static __constant__ float kSin32[16] = {
    0.f, 0x1.8f8b840000000p-3f, 0x1.87de2a0000000p-2f, 0x1.1c73b40000000p-1f,
    0x1.6a09e60000000p-1f, 0x1.a9b6620000000p-1f, 0x1.d906bc0000000p-1f, 0x1.f6297c0000000p-1f,
    0x1.0000000000000p+0f, 0x1.f6297c0000000p-1f, 0x1.d906bc0000000p-1f, 0x1.a9b6620000000p-1f,
    0x1.6a09e60000000p-1f, 0x1.1c73b40000000p-1f, 0x1.87de2a0000000p-2f, 0x1.8f8b840000000p-3f};

// One window of one interferogram. Rows of 34 floats: a lane reads its own row in
// 8-byte accesses and writes a column, both without bank conflicts; the pad
// staggers the tiles of a block's warps, so that its interleaved loads (all
// interferograms of one cell at once) hit distinct banks: 4 floats for 8 tiles a
// block, 8 for 4.
constexpr int kTileRow = 34;
template <int PAD>
struct ClapTileF {
  float re[32][kTileRow];
  float im[32][kTileRow];
  float hs[32][kTileRow];
  float pad[PAD];
};

enum FftPass : int {
  kForward1 = 0,  // own row of the zero-padded window; result transposed
  kForward2 = 1,  // own column of the spectrum; result and (transposed) magnitude
  kInverse1 = 2,  // gain from hs, re and im exchanged; result transposed
  kInverse2 = 3,  // own row; the result times the pyramid weights
  // the gradient's (FORM 2): without magnitude, gain and weights
  kForward2Plain = 4,
  kInverse1Plain = 5,
  kInverse2Plain = 6,
};

// The 32-point transform of lane's row of T; pass p of the window (uniform).
// Window rows and columns >= NZ are zero and, in pass 0, not read. In pass
// kInverse2 the lane's result times its pyramid weights wt[l] (l < nw) goes back to
// its row.
// FORM 0: all four passes; 1: the forward ones (adjoint's window); 2: the plain ones.
template <int NZ, int FORM, typename Tile>
__device__ __forceinline__ void fft_row_inline(Tile& T, const int lane, const int p, const float* wt, const int rs,
                                               const int cs, const int nw) {
  float2 ar[16], ai[16];  // points 2 m and 2 m + 1 at the bit reversal of m
  auto at = [](int m) { return ((m & 1) << 3) | ((m & 2) << 1) | ((m & 4) >> 1) | ((m & 8) >> 3); };
  if (p == kForward1) {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = at(m);
      ar[j] = ai[j] = make_float2(0.f, 0.f);
      if (2 * m < NZ && lane < NZ) {
        ar[j] = *reinterpret_cast<const float2*>(&T.re[lane][2 * m]);
        ai[j] = *reinterpret_cast<const float2*>(&T.im[lane][2 * m]);
      }
    }
  } else if (FORM != 1 && p == (FORM == 0 ? kInverse1 : kInverse1Plain)) {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = at(m);
      ar[j] = *reinterpret_cast<const float2*>(&T.im[lane][2 * m]);
      ai[j] = *reinterpret_cast<const float2*>(&T.re[lane][2 * m]);
      if constexpr (FORM == 0) {
        const float2 g = *reinterpret_cast<const float2*>(&T.hs[lane][2 * m]);
        ar[j] = __fmul2_rn(ar[j], g);
        ai[j] = __fmul2_rn(ai[j], g);
      }
    }
  } else {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = at(m);
      ar[j] = *reinterpret_cast<const float2*>(&T.re[lane][2 * m]);
      ai[j] = *reinterpret_cast<const float2*>(&T.im[lane][2 * m]);
    }
  }
#pragma unroll
  for (int half = 1; half < 16; half <<= 1) {
    const int step = 16 / half;
#pragma unroll
    for (int s = 0; s < 16; s += 2 * half) {
#pragma unroll
      for (int k = 0; k < half; ++k) {
        const int ti = k * step, q = s + k + half;
        const float2 ur = ar[s + k], ui = ai[s + k], vr = ar[q], vi = ai[q];
        if (ti == 8) {  // t = -i v
          ar[s + k] = __fadd2_rn(ur, vi);
          ai[s + k] = sub2(ui, vr);
          ar[q] = sub2(ur, vi);
          ai[q] = __fadd2_rn(ui, vr);
        } else {
          float2 tr = vr, tj = vi;
          if (ti != 0) {
            const float2 wx = both(kCos32[ti]), ws = both(kSin32[ti]), nws = both(-kSin32[ti]);
            tr = __ffma2_rn(vr, wx, __fmul2_rn(vi, ws));   // factor cos - i sin
            tj = __ffma2_rn(vi, wx, __fmul2_rn(vr, nws));
          }
          ar[s + k] = __fadd2_rn(ur, tr);
          ai[s + k] = __fadd2_rn(ui, tj);
          ar[q] = sub2(ur, tr);
          ai[q] = sub2(ui, tj);
        }
      }
    }
  }
  // stage 5: point k of the even and of the odd half
  float xr[32], xi[32];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float ur = ar[k].x, ui = ai[k].x, vr = ar[k].y, vi = ai[k].y;
    float tr = vr, tj = vi;
    if (k == 8) {
      tr = vi;
      tj = -vr;
    } else if (k != 0) {
      tr = __fmaf_rn(vr, kCos32[k], __fmul_rn(vi, kSin32[k]));
      tj = __fmaf_rn(vi, kCos32[k], __fmul_rn(vr, -kSin32[k]));
    }
    xr[k] = __fadd_rn(ur, tr);
    xi[k] = __fadd_rn(ui, tj);
    xr[k + 16] = __fsub_rn(ur, tr);
    xi[k + 16] = __fsub_rn(ui, tj);
  }
  if (FORM != 2 && p == kForward2) {
    if constexpr (FORM != 2) {
      uint32_t far = 0;
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        const float2 r = make_float2(xr[k], xr[k + 1]), i = make_float2(xi[k], xi[k + 1]);
        *reinterpret_cast<float2*>(&T.re[lane][k]) = r;
        *reinterpret_cast<float2*>(&T.im[lane][k]) = i;
        const float2 q = __ffma2_rn(r, r, __fmul2_rn(i, i));
        const float2 m = sqrt_newton2(q);
        T.hs[k][lane] = m.x;
        T.hs[k + 1][lane] = m.y;
        far = max(far, max(__float_as_uint(q.x) - kSqrtLo, __float_as_uint(q.y) - kSqrtLo));
      }
      if (far >= kSqrtSpan) {  // a zero, a tiny or an infinite value among them
#pragma unroll 1
        for (int k = 0; k < 32; ++k)
          T.hs[k][lane] = sqrtf(__fmaf_rn(T.re[lane][k], T.re[lane][k], __fmul_rn(T.im[lane][k], T.im[lane][k])));
      }
    }
  } else if (FORM == 0 && p == kInverse2) {
    if (lane < nw) {
      const bool row_zero = lane < rs;
#pragma unroll
      for (int l = 0; l < NZ; l += 2) {
        const float2 wv = make_float2((row_zero || l < cs || l >= nw) ? 0.f : wt[l],
                                      (row_zero || l + 1 < cs || l + 1 >= nw) ? 0.f : wt[l + 1]);
        *reinterpret_cast<float2*>(&T.re[lane][l]) = __fmul2_rn(make_float2(xr[l], xr[l + 1]), wv);
        *reinterpret_cast<float2*>(&T.im[lane][l]) = __fmul2_rn(make_float2(xi[l], xi[l + 1]), wv);
      }
    }
  } else if (FORM == 2 && (p == kForward2Plain || p == kInverse2Plain)) {
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
      *reinterpret_cast<float2*>(&T.re[lane][k]) = make_float2(xr[k], xr[k + 1]);
      *reinterpret_cast<float2*>(&T.im[lane][k]) = make_float2(xi[k], xi[k + 1]);
    }
  } else {
    __syncwarp();  // every lane has read its row
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      if (k < NZ || p == kForward1) {
        T.re[k][lane] = xr[k];
        T.im[k][lane] = xi[k];
      }
    }
  }
  __syncwarp();
}

// The same out of line: the window kernels keep more registers live around it and
// are faster so (256 x 256 cells x 60 ifg: 1194 against 1335 us an iteration).
template <int NZ, int FORM = 0, typename Tile>
__device__ __noinline__ void fft_row(Tile& T, const int lane, const int p, const float* wt, const int rs, const int cs,
                                     const int nw) {
  fft_row_inline<NZ, FORM>(T, lane, p, wt, rs, cs, nw);
}

// The 7-tap smoothing of 32 values along an axis of the fftshifted spectrum: in
// unshifted coordinates a circular convolution cut at the Nyquist seam (neighbour
// k + d counts iff 0 <= ((k + 16) mod 32) + d < 32); taps in order, two outputs to
// a packed value, a tap across the seam adding 0.
__device__ __forceinline__ void smooth32(const float (&h)[32], const float (&g)[4], float (&o)[32]) {
#pragma unroll
  for (int k = 0; k < 32; k += 2) {
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int d = -3; d <= 3; ++d) {
      const int s0 = ((k + 16) & 31) + d, s1 = ((k + 17) & 31) + d;
      const bool v0 = s0 >= 0 && s0 < 32, v1 = s1 >= 0 && s1 < 32;
      const float2 x = make_float2(v0 ? h[(k + d) & 31] : 0.f, v1 ? h[(k + 1 + d) & 31] : 0.f);
      if (v0 || v1) acc = __ffma2_rn(x, both(g[d < 0 ? d + 3 : 3 - d]), acc);
    }
    o[k] = acc.x;
    o[k + 1] = acc.y;
  }
}

// |X| in hs (row = row frequency) -> the smoothed magnitude of lane's column,
// smoothed along the rows first (a lane its own row), then along the column.
template <typename Tile>
__device__ __forceinline__ void smooth_tile(Tile& T, const int lane, const float (&g)[4], float (&o)[32]) {
  float h[32];
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    const float2 v = *reinterpret_cast<const float2*>(&T.hs[lane][c]);
    h[c] = v.x;
    h[c + 1] = v.y;
  }
  smooth32(h, g, o);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 32; ++c) T.hs[c][lane] = o[c];
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    const float2 v = *reinterpret_cast<const float2*>(&T.hs[lane][c]);
    h[c] = v.x;
    h[c + 1] = v.y;
  }
  smooth32(h, g, o);
}

// The 512th and 513th smallest of the 1,024 non-negative values held 32 per lane,
// exact (median(), native_stage2.rs:1173-1184, is their mean). A bracket of IEEE
// bit patterns (which order non-negative floats like their values) around the
// 512th is narrowed until it holds at most 32 values, which are then ranked among
// themselves in `scratch` (32 floats of the warp's). The pivot aims, on the line
// through the bracket's counts, a few ranks beyond the 512th on the side that was
// cut last from the other, so that both ends close in; every fourth pivot halves.
__device__ __forceinline__ void median_pair1024(const float (&o)[32], float* scratch, float& v0, float& v1) {
  const int lane = threadIdx.x & 31;
  uint32_t lo4[4], hi4[4];  // four chains each: their latencies overlap
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const uint32_t u = __float_as_uint(o[i]);
    lo4[i & 3] = i < 4 ? u : min(lo4[i & 3], u);
    hi4[i & 3] = i < 4 ? u : max(hi4[i & 3], u);
  }
  uint32_t lo = __reduce_min_sync(kFull, min(min(lo4[0], lo4[1]), min(lo4[2], lo4[3])));
  uint32_t hi = __reduce_max_sync(kFull, max(max(hi4[0], hi4[1]), max(hi4[2], hi4[3])));
  int cnt_lo = 0, cnt_hi = 1024;  // values below lo, values up to hi
  float aim = 512.f;
  int pass = 0;
  while (lo < hi && cnt_hi - cnt_lo > 32) {
    const uint32_t width = hi - lo;
    uint32_t step = width >> 1;
    if ((++pass & 3) != 0) {
      const float f = (aim - static_cast<float>(cnt_lo)) / static_cast<float>(cnt_hi - cnt_lo);
      step = static_cast<uint32_t>(static_cast<float>(width) * fminf(fmaxf(f, 0.f), 1.f));
      step = min(step, width - 1);
    }
    const uint32_t mid = lo + step;
    unsigned c4[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < 32; ++i) c4[i & 3] += (__float_as_uint(o[i]) <= mid) ? 1u : 0u;
    const unsigned cnt = __reduce_add_sync(kFull, (c4[0] + c4[1]) + (c4[2] + c4[3]));
    if (cnt >= 512u) {
      hi = mid;
      cnt_hi = static_cast<int>(cnt);
      aim = 512.f - 12.f;
    } else {
      lo = mid + 1;
      cnt_lo = static_cast<int>(cnt);
      aim = 512.f + 12.f;
    }
  }
  const int r0 = 511 - cnt_lo;  // rank of the 512th smallest inside the bracket
  bool next = false;            // the 513th is the smallest value above the bracket
  if (lo == hi) {
    v0 = v1 = __uint_as_float(lo);
    next = cnt_hi < 513;
  } else {
    const uint32_t width = hi - lo;
    int m4[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 32; ++i) m4[i & 3] += (__float_as_uint(o[i]) - lo <= width) ? 1 : 0;
    const int mine = (m4[0] + m4[1]) + (m4[2] + m4[3]);
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += t;
    }
    int off = incl - mine;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (__float_as_uint(o[i]) - lo <= width) scratch[off++] = o[i];
    __syncwarp();
    const int nb = cnt_hi - cnt_lo;
    const float x = lane < nb ? scratch[lane] : 0.f;
    int rank = 0;
    for (int j = 0; j < nb; ++j) {
      const float y = scratch[j];
      rank += (y < x || (y == x && j < lane)) ? 1 : 0;
    }
    const unsigned m0 = __ballot_sync(kFull, lane < nb && rank == r0);
    const unsigned m1 = __ballot_sync(kFull, lane < nb && rank == r0 + 1);
    v0 = __shfl_sync(kFull, x, __ffs(m0) - 1);
    v1 = __shfl_sync(kFull, x, __ffs(m1) - 1);
    next = r0 + 1 >= nb;
  }
  if (next) {
    uint32_t nxt = ~0u;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const uint32_t u = __float_as_uint(o[i]);
      if (u > hi) nxt = min(nxt, u);
    }
    v1 = __uint_as_float(__reduce_min_sync(kFull, nxt));
  }
  __syncwarp();
}

// Gain of lane's column, gk[k] = max((o[k] / med)^alpha - 1, 0) beta + low pass, to
// the lane's row of hs.
template <typename Tile>
__device__ __forceinline__ void gain_tile(Tile& T, const int lane, const float (&o)[32], const float med,
                                          const int alpha_is_one, const float alpha, const float beta,
                                          const float* lp) {
  const float inv_med = med != 0.f ? 1.f / med : 1.f;
#pragma unroll
  for (int k = 0; k < 32; k += 2) {
    float g[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float v = __fmul_rn(o[k + e], inv_med);
      v = __fadd_rn(alpha_is_one ? v : powf(v, alpha), -1.f);
      if (v < 0.f) v = 0.f;
      g[e] = __fmaf_rn(v, beta, lp[(k + e) * 32 + lane]);
    }
    *reinterpret_cast<float2*>(&T.hs[lane][k]) = make_float2(g[0], g[1]);
  }
}

}  // namespace ps2
