// The FP32 topofit: one patch's rows and a batch's.
#include <stdint.h>

#include <algorithm>
#include <cstdlib>

#include "phase_math.cuh"
#include "ps2_device.cuh"
#include "ps2_kernels.cuh"
#include "trial_interp_taps.h"

namespace ps2 {

cudaError_t kernel_attributes_once(size_t dynamic_smem);

// One group of L lanes per PS (L = 4, 8, 16 or 32, chosen from the number of
// interferograms so a lane owns about 5-10 columns); a warp holds 32/L PS.
// Column data (psdph z_c, the per-step rotation, bp_c) live in shared memory.
// The trial sweep finds the first argmax over the trials of |S_m|,
//   S_m = sum_c z_c e^{-j theta_c m},  theta_c = bp_c / range * pi/4,
// 16 magnitudes |m| at a time with the trial pairs +-m sharing one phasor
// chain, two trials per packed FP32x2 value, the chain started exactly in the
// middle of the block and run both ways by the three-term recurrence; the group
// then reduces its partial sums with a transposing butterfly. For n_half in
// 41 .. 87 it is sampled (sampled_sweep): the centred sum is evaluated at every
// 4th trial and interpolated between; otherwise every magnitude is swept
// (sweep_trial_pairs).

constexpr float kQuarterPiF = 3.14159265358979323846f / 4.0f;  // Rust std::f32::consts::PI / 4.0

// e^{-j x} for the re-anchoring points, |x| < ~1e3: Cody-Waite argument
// reduction by 2 pi with a two-constant split of 2 pi (Cody & Waite, "Software
// Manual for the Elementary Functions", 1980) to |r| <= pi, then the hardware
// sin/cos approximations (absolute error ~4e-7 on that range; a reduction to
// pi/4 with a quadrant rotation buys no accuracy there and costs a conversion
// and four selects per call).
__device__ __forceinline__ float2 cis_neg_anchor(float x) {
  const float k = rintf(x * 0.159154943091895335769f);
  float r = fmaf(-k, 6.28318548202514648438f, x);
  r = fmaf(-k, -1.74845553146951715e-7f, r);
  return make_float2(__cosf(r), -__sinf(r));
}

template <int L>
__device__ __forceinline__ float group_min(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
template <int L>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// |v|^2 with its rounding fixed: the trials of a row are ranked by it, and left to
// the compiler the product that joins the FMA differs from kernel to kernel (a tie
// of one row in 200,000 then goes another way in a batch than alone).
__device__ __forceinline__ float square(const float2 v) { return __fmaf_rn(v.x, v.x, __fmul_rn(v.y, v.y)); }

// Sum over the L lanes of a group of each of the W slots of v. Halving steps
// (lanes whose offset bit is set keep the upper half) while more than one slot
// remains, plain xor reductions after that. Returns the number of slots the
// lane holds (max(W/L, 1)) in v[0..]; they are slots base .. base+count-1.
template <int W, int L>
__device__ __forceinline__ int group_transpose_reduce(float2 (&v)[W], const int gl, int& base) {
  int cnt = W;
  base = 0;
#pragma unroll
  for (int o = L / 2; o >= 1; o >>= 1) {
    if (cnt > 1) {
      const int h = cnt / 2;
      const bool upper = (gl & o) != 0;
#pragma unroll
      for (int i = 0; i < W / 2; ++i) {
        if (i < h) {
          const float2 lo = v[i], hi = v[i + h];
          float2 send = upper ? lo : hi;
          const float2 keep = upper ? hi : lo;
          send.x = __shfl_xor_sync(kFull, send.x, o);
          send.y = __shfl_xor_sync(kFull, send.y, o);
          v[i] = make_float2(keep.x + send.x, keep.y + send.y);
        }
      }
      if (upper) base += h;
      cnt = h;
    } else {
      v[0].x += __shfl_xor_sync(kFull, v[0].x, o);
      v[0].y += __shfl_xor_sync(kFull, v[0].y, o);
    }
  }
  return cnt;
}

// Per-PS column store: z (psdph), e^{-j theta} (the per-trial rotation, theta =
// bp/range*pi/4 as the reference rounds it) and bp. Anchor angles are formed as
// bp * ((pi/4)/range) * m. Complex values lie together: one 8-byte access for two.
struct ColumnSmem {
  float2 *z, *r;
  float* bp;
};

// Trials +m and -m from one rotation chain, two columns per packed FP32x2
// instruction (the form of the last, odd magnitude of a sweep; the blocks of
// 2-16 magnitudes pack two trials instead, sweep_trial_pairs). For a column z = (x, y) and w = e^{-j m theta}:
//   z w       = (x w.x - y w.y, x w.y + y w.x)               trial +m
//   z conj(w) = (x w.x + y w.y, y w.x - x w.y) = z e^{+j m theta}   trial -m
// so the four sums  sum x w.x, sum x w.y, sum y w.y, sum y w.x  give both
// trials. A lane holds its columns in pairs (c0, c1) = (gl + L k, gl + L (k+1)):
// Wx = (w0.x, w1.x), Wy = (w0.y, w1.y) and the accumulators are FP32x2 pairs
// (one column of the pair in each half), added together once per block. One
// |m| step is then 4 packed instructions for the rotation
//   Wx <- Wx Rx - Wy Ry,  Wy <- Wx Ry + Wy Rx      (R = e^{-j theta})
// and 4 for the sums, i.e. 1 instruction per (trial, column). w is re-anchored
// exactly (cis_neg_anchor of theta * m) at the first |m| of every block, so a
// chain is at most W - 1 rotations long.
struct PackedCols {
  float2 x, y, rx, ry, nry, wx, wy;
};

// c1 < 0: no second column (its terms are zero)
__device__ __forceinline__ PackedCols load_packed_cols(const ColumnSmem& cs, const int c0, const int c1_or_none,
                                                       const float qr, const int m0) {
  PackedCols p;
  const int c1 = c1_or_none < 0 ? c0 : c1_or_none;
  const float2 z0 = cs.z[c0], z1 = c1_or_none < 0 ? make_float2(0.f, 0.f) : cs.z[c1], r0 = cs.r[c0], r1 = cs.r[c1];
  p.x = make_float2(z0.x, z1.x);
  p.y = make_float2(z0.y, z1.y);
  p.rx = make_float2(r0.x, r1.x);
  p.ry = make_float2(r0.y, r1.y);
  p.nry = make_float2(-p.ry.x, -p.ry.y);
  const float2 w0 = cis_neg_anchor(cs.bp[c0] * qr * static_cast<float>(m0));
  const float2 w1 = cis_neg_anchor(cs.bp[c1] * qr * static_cast<float>(m0));
  p.wx = make_float2(w0.x, w1.x);
  p.wy = make_float2(w0.y, w1.y);
  return p;
}

template <int W>
__device__ __forceinline__ void accumulate_packed(float2 (&Axx)[W], float2 (&Axy)[W], float2 (&Ayy)[W],
                                                  float2 (&Ayx)[W], PackedCols& p, const int k) {
  Axx[k] = __ffma2_rn(p.x, p.wx, Axx[k]);
  Axy[k] = __ffma2_rn(p.x, p.wy, Axy[k]);
  Ayy[k] = __ffma2_rn(p.y, p.wy, Ayy[k]);
  Ayx[k] = __ffma2_rn(p.y, p.wx, Ayx[k]);
  if (k + 1 < W) {
    const float2 t = __fmul2_rn(p.wy, p.nry);
    const float2 u = __fmul2_rn(p.wy, p.rx);
    const float2 wx = p.wx;
    p.wx = __ffma2_rn(wx, p.rx, t);
    p.wy = __ffma2_rn(wx, p.ry, u);
  }
}

// One block of W trial pairs |m| = m0 .. m0+W-1 (m0 >= 1): trial indices
// n_half + m and n_half - m. The running best
// keeps the first maximum in trial order (argmax_first_f32, :1526-1536)
// although the trials arrive out of order.
template <int W, int L>
__device__ __forceinline__ void sweep_pairs(const ColumnSmem& cs, const float qr, const int ncl, const int gl,
                                            const int m0, const int n_half, float& best_sq, int& best_t) {
  float2 Axx[W], Axy[W], Ayy[W], Ayx[W];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    Axx[k] = make_float2(0.f, 0.f);
    Axy[k] = make_float2(0.f, 0.f);
    Ayy[k] = make_float2(0.f, 0.f);
    Ayx[k] = make_float2(0.f, 0.f);
  }
  int k = 0;
  for (; k + 3 < ncl; k += 4) {
    PackedCols p0 = load_packed_cols(cs, gl + L * k, gl + L * (k + 1), qr, m0);
    PackedCols p1 = load_packed_cols(cs, gl + L * (k + 2), gl + L * (k + 3), qr, m0);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      accumulate_packed<W>(Axx, Axy, Ayy, Ayx, p0, j);
      accumulate_packed<W>(Axx, Axy, Ayy, Ayx, p1, j);
    }
  }
  for (; k < ncl; k += 2) {
    PackedCols p0 = load_packed_cols(cs, gl + L * k, k + 1 < ncl ? gl + L * (k + 1) : -1, qr, m0);
#pragma unroll
    for (int j = 0; j < W; ++j) accumulate_packed<W>(Axx, Axy, Ayy, Ayx, p0, j);
  }
  float2 S[2 * W];
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const float xx = Axx[j].x + Axx[j].y, xy = Axy[j].x + Axy[j].y;
    const float yy = Ayy[j].x + Ayy[j].y, yx = Ayx[j].x + Ayx[j].y;
    S[j] = make_float2(xx - yy, xy + yx);
    S[W + j] = make_float2(xx + yy, yx - xy);
  }
  int base;
  const int cnt = group_transpose_reduce<2 * W, L>(S, gl, base);
#pragma unroll
  for (int j = 0; j < (2 * W / L > 1 ? 2 * W / L : 1); ++j) {
    if (j < cnt) {
      const int idx = base + j;
      const int t = idx < W ? n_half + m0 + idx : n_half - (m0 + idx - W);
      const float sq = square(S[j]);
      if (sq > best_sq || (sq == best_sq && t < best_t)) {
        best_sq = sq;
        best_t = t;
      }
    }
  }
}

// One block of W trial magnitudes |m| = m0 .. m0+W-1 (W even, m0 >= 1) with
// two TRIALS per packed FP32x2 value: slot i of each accumulator holds
// (|m| = m0+2i, m0+2i+1), so W trial pairs cost 2W accumulator registers and
// one exact anchor per column covers all W magnitudes. Per column, with
// A = H/2 - 1 the middle slot: w(m0+2A) = e^{-j (m0+2A) theta} exactly,
// w(m0+2A+1) = w(m0+2A) e^{-j theta}, the next pair by one complex multiply with
// e^{-2j theta}, and every other pair, up and down from there, by the
// three-term recurrence of cos and sin (Chebyshev):
//   w(m+2) = 2 cos(2 theta) w(m) - w(m-2),   w(m-2) = 2 cos(2 theta) w(m) - w(m+2),
// one packed FMA per component instead of a complex multiply. It is carried as
// u_i = s_i w(m0+2i) with the sign pattern s_{A+j} = +,+,-,-,+,+,... (j mod 4)
// so that each step is a plain FMA (C = 2 cos 2theta):
//   u_{i+1} = ((i-A) odd ? -C : C) u_i + u_{i-1},  u_{i-1} = u_{i+1} - ((i-A) odd ? -C : C) u_i;
// the slot's sums then carry the factor s_i, which |S|^2 does not see.
// An error e in the two starting pairs grows to at most (k+1) e after k steps
// (|U_k(cos phi)| = |sin (k+1) phi / sin phi| <= k+1); starting in the middle
// keeps k <= H/2, so the phasor error stays near 2e-6 for H = 8 (1.4e-6 for a
// chain of complex multiplies), against 5.5e-6 for a chain started at slot 0.
// The four sums P = sum x w.x, Q = sum x w.y, R = sum y w.x, U = sum y w.y give
// S(+m) = (P - U, Q + R) and S(-m) = (P + U, R - Q) for both trials of a slot
// (up to the common sign s_i). Each lane sums its columns in column order; the
// group joins its lanes with the transposing reduction.
template <int W, int L>
__device__ __forceinline__ void sweep_trial_pairs(const ColumnSmem& cs, const float qr, const int ncl, const int gl,
                                                  const int m0, const int n_half, float& best_sq, int& best_t) {
  constexpr int H = W / 2;
  float2 P[H], Q[H], R[H], U[H];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    P[i] = make_float2(0.f, 0.f);
    Q[i] = make_float2(0.f, 0.f);
    R[i] = make_float2(0.f, 0.f);
    U[i] = make_float2(0.f, 0.f);
  }
#pragma unroll 2
  for (int k = 0; k < ncl; ++k) {
    const int c = gl + L * k;
    const float2 z = cs.z[c], r = cs.r[c];
    const float x = z.x, y = z.y, rx = r.x, ry = r.y;
    // the chain starts at slot A (the middle of the block) and runs both ways
    constexpr int A = H > 1 ? H / 2 - 1 : 0;
    const float2 a0 = cis_neg_anchor(cs.bp[c] * qr * static_cast<float>(m0 + 2 * A));
    const float a1x = fmaf(a0.x, rx, -a0.y * ry), a1y = fmaf(a0.x, ry, a0.y * rx);
    const float r2x = fmaf(rx, rx, -ry * ry), r2y = 2.f * rx * ry;
    const float2 X = make_float2(x, x), Y = make_float2(y, y);
    const float2 Cp = make_float2(2.f * r2x, 2.f * r2x), Cn = make_float2(-2.f * r2x, -2.f * r2x);
    // u_A = (w(m0+2A), w(m0+2A+1)), u_{A+1} = u_A e^{-2j theta}
    const float2 UAx = make_float2(a0.x, a1x), UAy = make_float2(a0.y, a1y);
    P[A] = __ffma2_rn(X, UAx, P[A]);
    Q[A] = __ffma2_rn(X, UAy, Q[A]);
    R[A] = __ffma2_rn(Y, UAx, R[A]);
    U[A] = __ffma2_rn(Y, UAy, U[A]);
    if (H > 1) {
      const float2 UBx = make_float2(fmaf(a0.x, r2x, -a0.y * r2y), fmaf(a1x, r2x, -a1y * r2y));
      const float2 UBy = make_float2(fmaf(a0.x, r2y, a0.y * r2x), fmaf(a1x, r2y, a1y * r2x));
      // forward: u_{i+1} = (i - A odd ? -C : C) u_i + u_{i-1}
      float2 Vx = UAx, Vy = UAy, Wx = UBx, Wy = UBy;
#pragma unroll
      for (int i = A + 1; i < H; ++i) {
        P[i] = __ffma2_rn(X, Wx, P[i]);
        Q[i] = __ffma2_rn(X, Wy, Q[i]);
        R[i] = __ffma2_rn(Y, Wx, R[i]);
        U[i] = __ffma2_rn(Y, Wy, U[i]);
        if (i + 1 < H) {
          const float2 nx = __ffma2_rn(((i - A) & 1) ? Cn : Cp, Wx, Vx);
          const float2 ny = __ffma2_rn(((i - A) & 1) ? Cn : Cp, Wy, Vy);
          Vx = Wx;
          Vy = Wy;
          Wx = nx;
          Wy = ny;
        }
      }
      // backward: u_{i-1} = u_{i+1} - (i - A odd ? -C : C) u_i
      Vx = UBx;
      Vy = UBy;
      Wx = UAx;
      Wy = UAy;
#pragma unroll
      for (int i = A; i > 0; --i) {
        const float2 nx = __ffma2_rn(((A - i) & 1) ? Cp : Cn, Wx, Vx);
        const float2 ny = __ffma2_rn(((A - i) & 1) ? Cp : Cn, Wy, Vy);
        Vx = Wx;
        Vy = Wy;
        Wx = nx;
        Wy = ny;
        P[i - 1] = __ffma2_rn(X, Wx, P[i - 1]);
        Q[i - 1] = __ffma2_rn(X, Wy, Q[i - 1]);
        R[i - 1] = __ffma2_rn(Y, Wx, R[i - 1]);
        U[i - 1] = __ffma2_rn(Y, Wy, U[i - 1]);
      }
    }
  }
  // slots 0..W-1: trials +m0..+m0+W-1; W..2W-1: trials -m0..-(m0+W-1)
  float2 S[2 * W];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    S[2 * i] = make_float2(P[i].x - U[i].x, Q[i].x + R[i].x);
    S[2 * i + 1] = make_float2(P[i].y - U[i].y, Q[i].y + R[i].y);
    S[W + 2 * i] = make_float2(P[i].x + U[i].x, R[i].x - Q[i].x);
    S[W + 2 * i + 1] = make_float2(P[i].y + U[i].y, R[i].y - Q[i].y);
  }
  int base;
  const int cnt = group_transpose_reduce<2 * W, L>(S, gl, base);
#pragma unroll
  for (int j = 0; j < (2 * W / L > 1 ? 2 * W / L : 1); ++j) {
    if (j < cnt) {
      const int idx = base + j;
      const int t = idx < W ? n_half + m0 + idx : n_half - (m0 + idx - W);
      const float sq = square(S[j]);
      if (sq > best_sq || (sq == best_sq && t < best_t)) {
        best_sq = sq;
        best_t = t;
      }
    }
  }
}

// ---- sampled trial sweep ---------------------------------------------------
// Only the argmax of |S_m|^2 over the trials leaves the sweep (the refinement
// recomputes K and the coherence exactly), and |S_m| = |T(m)| for the trial sum
// centred on the middle of the PS's bperp range,
//   T(m) = sum_c z_c e^{-j phi_c m},  phi_c = (bp_c - mid) (pi/4) / range,
// whose phases span exactly [-pi/8, pi/8]: T is band-limited to a quarter of
// the trial rate. It is evaluated exactly (same recurrences as the full sweep)
// at every 4th trial, m = 4k for |k| <= 16 NB, and between the samples by
// 20-tap fractional-delay filters (trial_interp_taps.h: error at most 6.8e-8 of
// sum |z_c|, below the FP32 rounding of the sums), so the sweep costs 16 NB + ~8
// magnitude steps instead of n_half. The samples stay in registers until the
// sweep ends (the column store's rotation slots, which the sample region
// overlays, are read until then).
constexpr int kMaxSampleBlocks = 2;

// Number of 16-magnitude sample blocks for n_half, or 0 where the full sweep
// is the cheaper (n_half <= 16 NB + 8) or the samples would exceed three blocks.
__host__ __device__ inline int trial_sample_blocks(int n_half) {
  const int ks = n_half / kTrialStride + (kInterpTapLo + kInterpTaps);  // floor(n/4) + 11 > the top tap
  const int nb = (ks + 15) / 16;
  if (nb < 2 || nb > kMaxSampleBlocks || 16 * nb + 8 >= n_half) return 0;
  return nb;
}

// Samples the filters read: T(4k) for k in [-kn, kp], kn = ceil(n/4) - tap_lo,
// kp = floor(n/4) + the top tap; kept at samp[kn + k].
__host__ __device__ inline int trial_samples_below(int n_half) { return (n_half + 3) / 4 - kInterpTapLo; }
__host__ __device__ inline int trial_samples_count(int n_half) {
  return trial_samples_below(n_half) + n_half / 4 + (kInterpTapLo + kInterpTaps - 1) + 1;
}

// Shared memory per PS in floats: a slot with z (2) and rotation (2) columns, with
// the sample array over the rotations when it fits there and after them otherwise,
// and a slot with the bp columns. The slots' strides put the groups of a warp on
// different banks: 2 L (mod 32) for the 8-byte accesses, which go by half warps, L
// for the 4-byte ones.
__host__ __device__ inline int topofit_sample_offset(int mpad, int n_half) {
  const int nb = trial_sample_blocks(n_half);
  return (nb == 0 || trial_samples_count(n_half) <= mpad) ? 2 * mpad : 4 * mpad;
}
__host__ __device__ inline int topofit_stride(int L, int mpad, int n_half) {
  const int nb = trial_sample_blocks(n_half);
  int need = 4 * mpad;
  if (nb > 0) {
    const int top = topofit_sample_offset(mpad, n_half) + 2 * trial_samples_count(n_half);
    need = top > need ? top : need;
  }
  return ((need - 2 * L + 31 + 64) / 32 - 2) * 32 + 2 * L;
}
__host__ __device__ inline int topofit_bp_stride(int L, int mpad) { return ((mpad - L + 31) / 32) * 32 + L; }

// One block of 16 sample magnitudes |k| = k0 .. k0+15 (the body of
// sweep_trial_pairs<16> with the centred phase per sample a_c = (bp_c - mid) qa
// and rotation e^{-j a_c} in the column store). Returns the lane's 32/L
// group-summed slots (slot idx < 16: T(4 (k0+idx)); else T(-4 (k0+idx-16))),
// the first of them at slot `base`.
template <int L>
__device__ __forceinline__ void sweep_sample_block(const ColumnSmem& cs, const float qa, const float mid,
                                                   const int ncl, const int gl, const int k0,
                                                   float2 (&out)[32 / L], int& base) {
  constexpr int H = 8;
  float2 P[H], Q[H], R[H], U[H];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    P[i] = make_float2(0.f, 0.f);
    Q[i] = make_float2(0.f, 0.f);
    R[i] = make_float2(0.f, 0.f);
    U[i] = make_float2(0.f, 0.f);
  }
#pragma unroll 3
  for (int k = 0; k < ncl; ++k) {
    const int c = gl + L * k;
    const float2 z = cs.z[c], r = cs.r[c];
    const float x = z.x, y = z.y, rx = r.x, ry = r.y;
    constexpr int A = H / 2 - 1;
    const float2 a0 = cis_neg_anchor((cs.bp[c] - mid) * qa * static_cast<float>(k0 + 2 * A));
    const float a1x = fmaf(a0.x, rx, -a0.y * ry), a1y = fmaf(a0.x, ry, a0.y * rx);
    const float r2x = fmaf(rx, rx, -ry * ry), r2y = 2.f * rx * ry;
    const float2 X = make_float2(x, x), Y = make_float2(y, y);
    const float2 Cp = make_float2(2.f * r2x, 2.f * r2x), Cn = make_float2(-2.f * r2x, -2.f * r2x);
    const float2 UAx = make_float2(a0.x, a1x), UAy = make_float2(a0.y, a1y);
    const float2 UBx = make_float2(fmaf(a0.x, r2x, -a0.y * r2y), fmaf(a1x, r2x, -a1y * r2y));
    const float2 UBy = make_float2(fmaf(a0.x, r2y, a0.y * r2x), fmaf(a1x, r2y, a1y * r2x));
    P[A] = __ffma2_rn(X, UAx, P[A]);
    Q[A] = __ffma2_rn(X, UAy, Q[A]);
    R[A] = __ffma2_rn(Y, UAx, R[A]);
    U[A] = __ffma2_rn(Y, UAy, U[A]);
    float2 Vx = UAx, Vy = UAy, Wx = UBx, Wy = UBy;
#pragma unroll
    for (int i = A + 1; i < H; ++i) {
      P[i] = __ffma2_rn(X, Wx, P[i]);
      Q[i] = __ffma2_rn(X, Wy, Q[i]);
      R[i] = __ffma2_rn(Y, Wx, R[i]);
      U[i] = __ffma2_rn(Y, Wy, U[i]);
      if (i + 1 < H) {
        const float2 nx = __ffma2_rn(((i - A) & 1) ? Cn : Cp, Wx, Vx);
        const float2 ny = __ffma2_rn(((i - A) & 1) ? Cn : Cp, Wy, Vy);
        Vx = Wx;
        Vy = Wy;
        Wx = nx;
        Wy = ny;
      }
    }
    Vx = UBx;
    Vy = UBy;
    Wx = UAx;
    Wy = UAy;
#pragma unroll
    for (int i = A; i > 0; --i) {
      const float2 nx = __ffma2_rn(((A - i) & 1) ? Cp : Cn, Wx, Vx);
      const float2 ny = __ffma2_rn(((A - i) & 1) ? Cp : Cn, Wy, Vy);
      Vx = Wx;
      Vy = Wy;
      Wx = nx;
      Wy = ny;
      P[i - 1] = __ffma2_rn(X, Wx, P[i - 1]);
      Q[i - 1] = __ffma2_rn(X, Wy, Q[i - 1]);
      R[i - 1] = __ffma2_rn(Y, Wx, R[i - 1]);
      U[i - 1] = __ffma2_rn(Y, Wy, U[i - 1]);
    }
  }
  // the chain's sign s_i is common to a slot's four sums: T itself carries it,
  // so undo it here (s_{A+j} = -1 for j mod 4 in {2, 3}; A = 3)
  float2 S[32];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const float s = (((i - 3) & 3) >= 2) ? -1.f : 1.f;
    S[2 * i] = make_float2(s * (P[i].x - U[i].x), s * (Q[i].x + R[i].x));
    S[2 * i + 1] = make_float2(s * (P[i].y - U[i].y), s * (Q[i].y + R[i].y));
    S[16 + 2 * i] = make_float2(s * (P[i].x + U[i].x), s * (R[i].x - Q[i].x));
    S[16 + 2 * i + 1] = make_float2(s * (P[i].y + U[i].y), s * (R[i].y - Q[i].y));
  }
  group_transpose_reduce<32, L>(S, gl, base);
#pragma unroll
  for (int j = 0; j < 32 / L; ++j) out[j] = S[j];
}

// Sampled sweep of a group: NB sample blocks, the samples the filters read
// written to `samp` (T(4k) at samp[kn + k]), then every trial t = n_half + m evaluated (exact
// at m = 4k, interpolated between) and the first maximum of |T|^2 kept in
// trial order. Lanes take chunks of 3 sample periods (12 trials) in turn and
// hold the 22 samples a chunk's filters read in registers.
template <int L, int NB>
__device__ __forceinline__ void sampled_sweep(const ColumnSmem& cs, float2* samp, const float qa, const float mid,
                                              const int ncl, const int gl, const int n_half, const float2 s0,
                                              float& best_sq, int& best_t) {
  constexpr int NO = 32 / L;
  const int kn = trial_samples_below(n_half), kp = trial_samples_count(n_half) - 1 - kn;
  float2 held[NB][NO];
  int bases[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) sweep_sample_block<L>(cs, qa, mid, ncl, gl, 1 + 16 * b, held[b], bases[b]);
  __syncwarp();  // every lane of the warp is done with the rotation columns
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int j = 0; j < NO; ++j) {
      const int idx = bases[b] + j;
      const int k = idx < 16 ? 1 + 16 * b + idx : -(1 + 16 * b + idx - 16);
      if (k >= -kn && k <= kp) samp[kn + k] = held[b][j];
    }
  }
  if (gl == 0) samp[kn] = s0;
  __syncwarp();
  constexpr int CP = 3, NWIN = CP + kInterpTaps - 1;
  const int klo = -((n_half + 3) / 4), khi = n_half / 4;  // floor(-n/4), floor(n/4)
  const int nch = (khi - klo + CP) / CP;
  best_sq = -1.f;
  best_t = 0x7fffffff;
  for (int ch = gl; ch < nch; ch += L) {
    const int kb = klo + ch * CP;
    float2 win[NWIN];  // T(4 (kb + kInterpTapLo + i))
#pragma unroll
    for (int i = 0; i < NWIN; ++i) {
      const int k = kb + kInterpTapLo + i;
      win[i] = (k >= -kn && k <= kp) ? samp[kn + k] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int pp = 0; pp < CP; ++pp) {
      const int k = kb + pp;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = 4 * k + r;
        float2 v;
        if (r == 0) {
          v = win[pp - kInterpTapLo];
        } else {
          v = make_float2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < kInterpTaps; ++i) {
            const float h = kInterpTaps_c[r - 1][i];
            v = __ffma2_rn(make_float2(h, h), win[pp + i], v);
          }
        }
        const float sq = square(v);
        const int t = n_half + m;
        if (m >= -n_half && m <= n_half && (sq > best_sq || (sq == best_sq && t < best_t))) {
          best_sq = sq;
          best_t = t;
        }
      }
    }
  }
}

// L2 prefetch of the rows a warp reads on its next pass (the PS group s0n ..
// s0n+G-1): the phase rows and, unless bperp is row invariant, the bperp rows,
// one 128-byte line per lane per instruction, all inside the arrays.
template <int G, bool ROWINV>
__device__ __forceinline__ void prefetch_rows(const void* ph, const float* bp, const int64_t s0n, const int64_t N,
                                              const int64_t M, const int lane) {
  if (s0n >= N) return;
  const int64_t s1 = s0n + G < N ? s0n + G : N;
  const char* p0 = static_cast<const char*>(ph) + s0n * M * 8;
  const int64_t nb = (s1 - s0n) * M * 8;
  for (int64_t o = static_cast<int64_t>(lane) * 128; o < nb; o += 32 * 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p0 + o));
  if (!ROWINV) {
    const char* b0 = reinterpret_cast<const char*>(bp + s0n * M);
    const int64_t nbb = (s1 - s0n) * M * 4;
    for (int64_t o = static_cast<int64_t>(lane) * 128; o < nbb; o += 32 * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(b0 + o));
  }
}

// The load step and the column store bound half of the kernel's instructions (2,550
// of 10,600 a warp pass at 150 interferograms before): columns come in pairs, z and
// the rotation lie as float2, magnitudes take sqrt_rn and columns are padded to the
// lanes only (152 for 150, not 160). 0.90 -> 0.81 ms at 250,000 PS x 150, 0.42 -> 0.38
// at 60, 0.21 -> 0.18 at 20 (81 trials); the same bits.
constexpr int kTopoLoadPairs = 4;  // the same in pairs of columns
constexpr int kTopoLoadCols = 8;  // columns whose loads a lane issues together in the prologue

// The work of block `vb` of a launch of `nvb` blocks over one patch: PS
// groups s0 = (vb * 4 + warp) * G + k * nvb * 4 * G. The batched kernel runs
// the same virtual blocks, so a patch's per-block rms partials, and with them
// its stop decisions, are the same as when it runs alone.
template <int L, bool LOOP, bool ROWINV>
__device__ __forceinline__ void topofit_vblock_t(const TopoArgs& a, const int mpad, const int vb, const int nvb,
                                                 unsigned char* smem_raw, int* sh_hist, double* sh_rms, int* sh_inv) {
  constexpr int G = 32 / L;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int g = lane / L, gl = lane % L;
  __syncthreads();
  for (int i = tid; i < kCohBins; i += blockDim.x) sh_hist[i] = 0;
  __syncthreads();
  const int stride = topofit_stride(L, mpad, a.n_half);
  float* base_ptr = reinterpret_cast<float*>(smem_raw) + static_cast<int64_t>(wib * G + g) * stride;
  const ColumnSmem cs{reinterpret_cast<float2*>(base_ptr), reinterpret_cast<float2*>(base_ptr) + mpad,
                      reinterpret_cast<float*>(smem_raw) + static_cast<int64_t>(4 * G) * stride +
                          static_cast<int64_t>(wib * G + g) * topofit_bp_stride(L, mpad)};
  const int nb = trial_sample_blocks(a.n_half);
  float2* samp = reinterpret_cast<float2*>(base_ptr + topofit_sample_offset(mpad, a.n_half));
  const float2* __restrict__ ph_nm = static_cast<const float2*>(a.ph_nm);
  const float2* __restrict__ filt = static_cast<const float2*>(a.filt);
  const float2* __restrict__ cpx = static_cast<const float2*>(a.cpx);
  float* __restrict__ K_out = static_cast<float*>(a.K_out);
  float* __restrict__ C_out = static_cast<float*>(a.C_out);
  float* __restrict__ coh_io = static_cast<float*>(a.coh_io);
  float2* __restrict__ resid = static_cast<float2*>(a.residual);
  float* __restrict__ ph_res = static_cast<float*>(a.ph_res);
  float2* __restrict__ ph_patch = static_cast<float2*>(a.ph_patch);
  const int64_t M = a.M;
  const int ncl = mpad / L;
  const unsigned gmask = (L == 32) ? kFull : (((1u << L) - 1u) << (g * L));
  double rms_acc = 0.0;
  int inv_acc = 0;
  const int64_t step = static_cast<int64_t>(nvb) * 4 * G;
  // the cell of this lane's next PS is loaded one pass ahead, so the
  // filtered-grid gather of a pass does not wait on it
  const int64_t s_first = (static_cast<int64_t>(vb) * 4 + wib) * G + g;
  int64_t cell_next = (LOOP && s_first < a.N) ? a.cell_of[s_first] : 0;
  for (int64_t s0 = (static_cast<int64_t>(vb) * 4 + wib) * G; s0 < a.N; s0 += step) {
    const int64_t s = s0 + g;
    const bool active = s < a.N;
    const int64_t cell = cell_next;
    if (LOOP) cell_next = s + step < a.N ? a.cell_of[s + step] : 0;
    prefetch_rows<G, ROWINV>(LOOP ? static_cast<const void*>(ph_nm) : static_cast<const void*>(cpx), a.bp, s0 + step,
                             a.N, M, lane);
    bool zero = false, nonzero = false;
    float mn = __int_as_float(0x7f800000), mx = -mn;
    if (LOOP && a.filt_unit && !ph_patch) {
      // two columns per round and lane, kTopoLoadPairs rounds' loads issued first: 16
      // bytes of patch phase and, for even M (rows then start on 16 bytes), of phase in
      // one access. A row with a zero element is invalid whatever its baselines, so
      // their extremes need no look at z.
      constexpr int PP = kTopoLoadPairs;
      const bool even = (a.M & 1) == 0;
      const int np = mpad / 2, mp = active ? (a.M + 1) / 2 : 0;
      const float4* __restrict__ f2 = reinterpret_cast<const float4*>(filt + cell * a.Mp);
      const float2* __restrict__ p1 = ph_nm + (active ? s : 0) * M;
      const float* __restrict__ b1 = ROWINV ? a.bp : a.bp + (active ? s : 0) * M;
      float least = 1.f;  // of max(|re z|, |im z|)
      for (int q0 = gl; q0 < np; q0 += PP * L) {
        float4 fv[PP], pv[PP];
        float2 bv[PP];
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          const int q = q0 + L * i;
          fv[i] = pv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          bv[i] = make_float2(0.f, 0.f);
          if (q < mp) {
            fv[i] = f2[q];
            if (even) {
              pv[i] = reinterpret_cast<const float4*>(p1)[q];
              bv[i] = reinterpret_cast<const float2*>(b1)[q];
            } else {
              const float2 x = p1[2 * q];
              pv[i].x = x.x;
              pv[i].y = x.y;
              bv[i].x = b1[2 * q];
              if (2 * q + 1 < a.M) {
                const float2 y = p1[2 * q + 1];
                pv[i].z = y.x;
                pv[i].w = y.y;
                bv[i].y = b1[2 * q + 1];
              }
            }
          }
        }
#pragma unroll
        for (int i = 0; i < PP; ++i) {
          const int q = q0 + L * i;
          if (q >= np) break;
          const float2 v0 = cmul_rn(make_float2(fv[i].x, -fv[i].y), make_float2(pv[i].x, pv[i].y));  // psdph (:687-689)
          const float2 v1 = cmul_rn(make_float2(fv[i].z, -fv[i].w), make_float2(pv[i].z, pv[i].w));
          if (q < mp) {
            least = fminf(least, fmaxf(fabsf(v0.x), fabsf(v0.y)));
            mn = fminf(mn, bv[i].x);
            mx = fmaxf(mx, bv[i].x);
            if (even || 2 * q + 1 < a.M) {
              least = fminf(least, fmaxf(fabsf(v1.x), fabsf(v1.y)));
              mn = fminf(mn, bv[i].y);
              mx = fmaxf(mx, bv[i].y);
            }
          }
          *reinterpret_cast<float4*>(&cs.z[2 * q]) = make_float4(v0.x, v0.y, v1.x, v1.y);
          *reinterpret_cast<float2*>(&cs.bp[2 * q]) = bv[i];
        }
      }
      zero = least == 0.f;
      nonzero = true;
      __syncwarp();  // the columns are read by other lanes of the group than stored them
    } else {
      // kTopoLoadCols columns per round with their global loads issued first
      constexpr int PR = kTopoLoadCols;
      for (int k0c = 0; k0c < ncl; k0c += PR) {
        float2 fv[PR], pv[PR];
        float bv[PR];
#pragma unroll
        for (int i = 0; i < PR; ++i) {
          const int c = gl + L * (k0c + i);
          fv[i] = make_float2(0.f, 0.f);
          pv[i] = make_float2(0.f, 0.f);
          bv[i] = 0.f;
          if (active && k0c + i < ncl && c < a.M) {
            if (!LOOP) {
              pv[i] = cpx[s * M + c];
            } else {
              fv[i] = filt[cell * a.Mp + c];
              pv[i] = ph_nm[s * M + c];
            }
            bv[i] = ROWINV ? a.bp[c] : a.bp[s * M + c];
          }
        }
#pragma unroll
        for (int i = 0; i < PR; ++i) {
          const int c = gl + L * (k0c + i);
          if (k0c + i >= ncl) break;
          float2 v = make_float2(0.f, 0.f);
          if (active && c < a.M) {
            if (!LOOP) {
              v = pv[i];
            } else {
              // extract_patch_phase + normalize_complex_unit_magnitude (:1186-1205)
              float2 f = fv[i];
              if (!a.filt_unit) {
                const float mag = hypotf(f.x, f.y);
                if (mag != 0.f) f = make_float2(f.x / mag, f.y / mag);
              }
              if (ph_patch) ph_patch[s * M + c] = f;
              v = cmul_rn(conjf2(f), pv[i]);  // psdph (:687-689)
            }
            if (v.x == 0.f && v.y == 0.f) {
              zero = true;
            } else {
              nonzero = true;
              mn = fminf(mn, bv[i]);
              mx = fmaxf(mx, bv[i]);
            }
          }
          cs.z[c] = v;
          cs.bp[c] = bv[i];
        }
      }
    }
    const bool any_zero = (__ballot_sync(kFull, zero) & gmask) != 0u;
    const bool any_nonzero = (__ballot_sync(kFull, nonzero) & gmask) != 0u;
    const bool invalid = !active || (a.zero_mode == 0 ? any_zero : !any_nonzero);
    mn = group_min<L>(mn);
    mx = group_max<L>(mx);
    float range = mx - mn;
    if (!(range != 0.f) || invalid) range = 1.f;
    // sampled sweep: rotation e^{-j a_c} per sample step, a_c = (bp_c - mid) qa;
    // full sweep: e^{-j theta_c} per trial, theta_c = bp_c / range * pi/4
    const float mid = (nb > 0 && !invalid && mx >= mn) ? 0.5f * (mn + mx) : 0.f;
    const float qa = (kQuarterPiF / range) * static_cast<float>(kTrialStride);
    for (int k = 0; k < ncl; ++k) {
      const int c = gl + L * k;
      const float t = nb > 0 ? (cs.bp[c] - mid) * qa : (cs.bp[c] / range) * kQuarterPiF;
      float sn, cn;
      sincos_cw(t, &sn, &cn);
      cs.r[c] = make_float2(cn, -sn);
    }
    const float qr = kQuarterPiF / range;
    __syncwarp();
    // trial sweep over m = -n .. n (all groups run it; invalid ones discard it):
    // m = 0 is the plain column sum, then the pairs +-m
    float best_sq, s0x = 0.f, s0y = 0.f;
    for (int k = 0; k < ncl; ++k) {
      const int c = gl + L * k;
      s0x += cs.z[c].x;
      s0y += cs.z[c].y;
    }
    s0x = group_sum<L>(s0x);
    s0y = group_sum<L>(s0y);
    best_sq = square(make_float2(s0x, s0y));
    int best_t = a.n_half;
    if (nb == 2) {
      sampled_sweep<L, 2>(cs, samp, qa, mid, ncl, gl, a.n_half, make_float2(s0x, s0y), best_sq, best_t);
    } else {
      int m0 = 1;
      for (; a.n_half - m0 + 1 >= 16; m0 += 16)
        sweep_trial_pairs<16, L>(cs, qr, ncl, gl, m0, a.n_half, best_sq, best_t);
      if (a.n_half - m0 + 1 >= 8) {
        sweep_trial_pairs<8, L>(cs, qr, ncl, gl, m0, a.n_half, best_sq, best_t);
        m0 += 8;
      }
      if (a.n_half - m0 + 1 >= 4) {
        sweep_trial_pairs<4, L>(cs, qr, ncl, gl, m0, a.n_half, best_sq, best_t);
        m0 += 4;
      }
      if (a.n_half - m0 + 1 >= 2) {
        sweep_trial_pairs<2, L>(cs, qr, ncl, gl, m0, a.n_half, best_sq, best_t);
        m0 += 2;
      }
      if (a.n_half - m0 + 1 >= 1) sweep_pairs<1, L>(cs, qr, ncl, gl, m0, a.n_half, best_sq, best_t);
    }
    // first maximum over the group (argmax_first_f32, :1526-1536)
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      const float osq = __shfl_xor_sync(kFull, best_sq, o);
      const int ot = __shfl_xor_sync(kFull, best_t, o);
      if (osq > best_sq || (osq == best_sq && ot < best_t)) {
        best_sq = osq;
        best_t = ot;
      }
    }
    if (best_t == 0x7fffffff) best_t = a.n_half;  // no finite |T|^2: the m = 0 trial, as the full sweep keeps
    __syncwarp();  // the sample array overlays the rotation slots written next
    // refine_candidate (:1259-1303) with FP64 normal-equation sums; the
    // rotation slots of the column store now hold z e^{-j k0 bp}
    const float k0 = kQuarterPiF / range * static_cast<float>(best_t - a.n_half);
    float ox = 0.f, oy = 0.f;
    for (int k = 0; k < ncl; ++k) {
      const int c = gl + L * k;
      const float2 r = cmul_rn(cs.z[c], cis_neg_anchor(k0 * cs.bp[c]));
      cs.r[c] = r;
      ox += r.x;
      oy += r.y;
    }
    ox = group_sum<L>(ox);
    oy = group_sum<L>(oy);
    const float2 oc = make_float2(ox, -oy);
    double mopt = 0.0, dl = 0.0;
    float den_w = 0.f;  // sum |z|: |residual| = |z| (a rotation), the refined coherence's denominator
    for (int k = 0; k < ncl; ++k) {
      const int c = gl + L * k;
      // in the loop |z| is that of a product of two unit (or zero) phasors, with
      // no overflow or underflow to guard against: sqrt(x^2 + y^2) is within an
      // ulp of hypotf at a third of its cost; standalone rows take any magnitude
      const float2 z = cs.z[c];
      const float wf = LOOP ? sqrt_rn(fmaf(z.x, z.x, z.y * z.y)) : hypotf(z.x, z.y);
      den_w += wf;
      const double wgt = static_cast<double>(wf);
      const double wb = __dmul_rn(wgt, static_cast<double>(cs.bp[c]));
      dl = __dadd_rn(dl, __dmul_rn(wb, wb));
      const float2 q = cmul_rn(cs.r[c], oc);
      mopt = __dadd_rn(mopt, __dmul_rn(wb, __dmul_rn(wgt, static_cast<double>(atan2_poly(q.y, q.x)))));
    }
    mopt = group_sum<L>(mopt);
    dl = group_sum<L>(dl);
    if (dl == 0.0) dl = 1.0;
    const float K1 = static_cast<float>(static_cast<double>(k0) + mopt / dl);
    float mx2 = 0.f, my2 = 0.f, den2 = den_w;
    for (int k = 0; k < ncl; ++k) {
      const int c = gl + L * k;
      const float2 r = cmul_rn(cs.z[c], cis_neg_anchor(K1 * cs.bp[c]));
      mx2 += r.x;
      my2 += r.y;
      if (active && c < a.M) {
        if (resid) resid[s * M + c] = invalid ? make_float2(0.f, 0.f) : r;
        if (ph_res) ph_res[s * M + c] = invalid ? 0.f : atan2f(r.y, r.x);
      }
    }
    mx2 = group_sum<L>(mx2);
    my2 = group_sum<L>(my2);
    den2 = group_sum<L>(den2);
    if (den2 == 0.f) den2 = 1.f;
    __syncwarp();
    if (gl == 0 && active) {
      float Kv, Cv, cohv;
      if (invalid) {
        // fit_stage2_rows invalid row (:676-697) / topofit_row empty row (:1216-1222)
        Kv = __int_as_float(0x7fffffff);
        Cv = a.zero_mode == 0 ? 0.f : Kv;
        cohv = a.zero_mode == 0 ? 0.f : Kv;
        inv_acc += 1;
      } else {
        Kv = K1;
        Cv = atan2f(my2, mx2);
        cohv = hypotf(mx2, my2) / den2;
      }
      if (a.accumulate_stats) {
        const double d = static_cast<double>(cohv) - static_cast<double>(coh_io[s]);
        rms_acc += d * d;
        const int b = coh_bin(static_cast<double>(cohv), a.cutoff0, a.dbin);
        if (b >= 0) atomicAdd(&sh_hist[b], 1);
      }
      K_out[s] = Kv;
      C_out[s] = Cv;
      coh_io[s] = cohv;
      if (a.nopt) a.nopt[s] = invalid ? 0 : 1;
    }
  }
  if (!a.accumulate_stats) return;
  rms_acc = warp_sum(rms_acc);
  inv_acc = warp_sum(inv_acc);
  if (lane == 0) {
    sh_rms[wib] = rms_acc;
    sh_inv[wib] = inv_acc;
  }
  __syncthreads();
  if (tid == 0) {
    a.rms_partial[vb] = sh_rms[0] + sh_rms[1] + sh_rms[2] + sh_rms[3];
    const int iv = sh_inv[0] + sh_inv[1] + sh_inv[2] + sh_inv[3];
    if (iv) atomicAdd(a.n_invalid, iv);
  }
  for (int i = tid; i < kCohBins; i += blockDim.x)
    if (sh_hist[i]) atomicAdd(&a.hist[i], sh_hist[i]);
}

// The input form (loop: ph_nm + filtered grid; standalone: psdph rows) and the
// row invariance of bperp are compile-time in the body.
template <int L>
__device__ __forceinline__ void topofit_vblock(const TopoArgs& a, const int mpad, const int vb, const int nvb,
                                               unsigned char* smem_raw, int* sh_hist, double* sh_rms, int* sh_inv) {
  if (a.cpx)
    a.bp_row_inv ? topofit_vblock_t<L, false, true>(a, mpad, vb, nvb, smem_raw, sh_hist, sh_rms, sh_inv)
                 : topofit_vblock_t<L, false, false>(a, mpad, vb, nvb, smem_raw, sh_hist, sh_rms, sh_inv);
  else
    a.bp_row_inv ? topofit_vblock_t<L, true, true>(a, mpad, vb, nvb, smem_raw, sh_hist, sh_rms, sh_inv)
                 : topofit_vblock_t<L, true, false>(a, mpad, vb, nvb, smem_raw, sh_hist, sh_rms, sh_inv);
}

template <int L>
__global__ void __launch_bounds__(128, 4) k_topofit_f32(TopoArgs a, int mpad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int sh_hist[kCohBins];
  __shared__ double sh_rms[4];
  __shared__ int sh_inv[4];
  topofit_vblock<L>(a, mpad, blockIdx.x, gridDim.x, smem_raw, sh_hist, sh_rms, sh_inv);
}

int topofit_lanes(int M) {
  static const int forced = [] {
    const char* e = getenv("PS2_TOPOFIT_LANES");
    return e ? atoi(e) : 0;
  }();
  if (forced == 4 || forced == 8 || forced == 16 || forced == 32) return forced;
  int L = 4;
  while (L < 32 && L * 24 < M) L *= 2;
  return L;
}

size_t topofit_smem_bytes(int L, int mpad, int n_half) {
  return static_cast<size_t>(4 * (32 / L)) * (topofit_stride(L, mpad, n_half) + topofit_bp_stride(L, mpad)) *
         sizeof(float);
}

// Columns per PS padded to a multiple of L (zero columns).
int topofit_mpad(int L, int M) { return ((M + L - 1) / L) * L; }

template <int L>
static cudaError_t topofit_geometry_l(const TopoArgs& a, int grid_cap, size_t* smem, int* blocks_out) {
  const int mpad = topofit_mpad(L, a.M);
  const size_t sm = topofit_smem_bytes(L, mpad, a.n_half);
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_topofit_f32<L>, 128, sm);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t per_block = 4 * (32 / L);
  int64_t blocks = (a.N + per_block - 1) / per_block;
  const int64_t cap = std::min<int64_t>(grid_cap, static_cast<int64_t>(sms) * std::max(per_sm, 1));
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  *smem = sm;
  *blocks_out = static_cast<int>(blocks);
  return cudaSuccess;
}

// Blocks of the FP32 topofit launch for this patch (the virtual blocks a batch
// reproduces); the lane count is a.lanes or the rule from M.
cudaError_t topofit_geometry(const TopoArgs& a, int grid_cap, int* L_out, int* mpad_out, int* blocks_out) {
  const int L = a.lanes ? a.lanes : topofit_lanes(a.M);
  size_t sm = 0;
  cudaError_t e;
  switch (L) {
    case 4: e = topofit_geometry_l<4>(a, grid_cap, &sm, blocks_out); break;
    case 8: e = topofit_geometry_l<8>(a, grid_cap, &sm, blocks_out); break;
    case 16: e = topofit_geometry_l<16>(a, grid_cap, &sm, blocks_out); break;
    case 32: e = topofit_geometry_l<32>(a, grid_cap, &sm, blocks_out); break;
    default: return cudaErrorInvalidValue;
  }
  *L_out = L;
  *mpad_out = topofit_mpad(L, a.M);
  return e;
}

template <int L>
static cudaError_t launch_topofit_l(const TopoArgs& a, int grid_cap, cudaStream_t st) {
  size_t sm = 0;
  int blocks = 0;
  cudaError_t e = topofit_geometry_l<L>(a, grid_cap, &sm, &blocks);
  if (e != cudaSuccess) return e;
  k_topofit_f32<L><<<static_cast<unsigned>(blocks), 128, sm, st>>>(a, topofit_mpad(L, a.M));
  return cudaGetLastError();
}

cudaError_t launch_topofit_f32(const TopoArgs& a, int grid_blocks, cudaStream_t st) {
  switch (a.lanes ? a.lanes : topofit_lanes(a.M)) {
    case 4: return launch_topofit_l<4>(a, grid_blocks, st);
    case 8: return launch_topofit_l<8>(a, grid_blocks, st);
    case 16: return launch_topofit_l<16>(a, grid_blocks, st);
    default: return launch_topofit_l<32>(a, grid_blocks, st);
  }
}

// ROWVAR: every patch of the batch has a bperp row per PS (one form of the body in
// the kernel: two spill).
template <int L, bool ROWVAR>
__global__ void __launch_bounds__(128, 4) k_batch_topofit(BatchArgs b, const int32_t* __restrict__ units, int n_units) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int sh_hist[kCohBins];
  __shared__ double sh_rms[4];
  __shared__ int sh_inv[4];
  for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
    const int p = units[2 * u], vb = units[2 * u + 1];
    if (!b.active[p]) continue;
    const PatchDev& d = b.patch[p];
    // batches hold loaded contexts: always the loop form
    if (!ROWVAR && d.topo.bp_row_inv)
      topofit_vblock_t<L, true, true>(d.topo, d.mpad, vb, d.nvb, smem_raw, sh_hist, sh_rms, sh_inv);
    else
      topofit_vblock_t<L, true, false>(d.topo, d.mpad, vb, d.nvb, smem_raw, sh_hist, sh_rms, sh_inv);
  }
}

template <int L, bool ROWVAR>
static cudaError_t batch_topofit_l(const BatchArgs& b, const int32_t* units, int n_units, size_t sm, int sm_count,
                                   cudaStream_t st) {
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_topofit<L, ROWVAR>, 128, sm);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min<int64_t>(n_units, static_cast<int64_t>(sm_count) * std::max(per_sm, 1));
  k_batch_topofit<L, ROWVAR><<<static_cast<unsigned>(blocks), 128, sm, st>>>(b, units, n_units);
  return cudaGetLastError();
}

template <bool ROWVAR>
static cudaError_t batch_topofit_form(const BatchArgs& b, int L, const int32_t* units, int n_units, size_t smem,
                                      int sm_count, cudaStream_t st) {
  switch (L) {
    case 4: return batch_topofit_l<4, ROWVAR>(b, units, n_units, smem, sm_count, st);
    case 8: return batch_topofit_l<8, ROWVAR>(b, units, n_units, smem, sm_count, st);
    case 16: return batch_topofit_l<16, ROWVAR>(b, units, n_units, smem, sm_count, st);
    case 32: return batch_topofit_l<32, ROWVAR>(b, units, n_units, smem, sm_count, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_batch_topofit(const BatchArgs& b, int L, const int32_t* units, int n_units, size_t smem, bool rowvar,
                                 int sm_count, cudaStream_t st) {
  if (n_units <= 0) return cudaSuccess;
  return rowvar ? batch_topofit_form<true>(b, L, units, n_units, smem, sm_count, st)
                : batch_topofit_form<false>(b, L, units, n_units, smem, sm_count, st);
}

cudaError_t topofit_f32_attributes(int optin) {
  const cudaError_t steps[] = {
      opt_in_smem(k_topofit_f32<4>, optin),    opt_in_smem(k_topofit_f32<8>, optin),
      opt_in_smem(k_topofit_f32<16>, optin),   opt_in_smem(k_topofit_f32<32>, optin),
      opt_in_smem(k_batch_topofit<4, false>, optin),  opt_in_smem(k_batch_topofit<4, true>, optin),
      opt_in_smem(k_batch_topofit<8, false>, optin),  opt_in_smem(k_batch_topofit<8, true>, optin),
      opt_in_smem(k_batch_topofit<16, false>, optin), opt_in_smem(k_batch_topofit<16, true>, optin),
      opt_in_smem(k_batch_topofit<32, false>, optin), opt_in_smem(k_batch_topofit<32, true>, optin),
  };
  for (const cudaError_t x : steps)
    if (x != cudaSuccess) return x;
  return cudaSuccess;
}

}  // namespace ps2
