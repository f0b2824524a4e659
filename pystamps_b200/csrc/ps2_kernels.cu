// Stage-2 gamma-estimation kernels for B200 (sm_100a).
//
// One iteration of the reference loop (crates/pystamps-core/src/native_stage2.rs:261-406)
// is six launches on one stream; the FP32 CLAP and topofit kernels are in
// clap_f32.cu and topofit_f32.cu, the others here:
//   k_iter_begin   state of the last iteration kept, P-square weights (:1674-1682)
//   k_bin          fill_phase_weight + accumulate_grid (:629-657, :722-740), fused,
//                  as a sort-by-cell sequential segmented reduction (no float atomics)
//   k_clap         clap_filter_one_ifg per (window, ifg) (:823-916): 32x32 FFT in
//                  registers + shared memory, |H| smoothing, median, filter, IFFT
//   k_overlap      the pyramid-weighted overlap-add (:904-915) as a gather in the
//                  reference's window order (deterministic), and the unit patch phase
//   k_topofit_f64  extract_patch_phase + fit_stage2_rows + topofit_row +
//                  refine_candidate (:1186-1303)
//   k_finalize     rms_difference, stop rule, P-square weighting table (:307-381, :1538-1783)
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "ps2_device.cuh"
#include "ps2_kernels.cuh"
#include "phase_math.cuh"

namespace ps2 {

cudaError_t kernel_attributes_once(size_t dynamic_smem);

template <typename R>
struct CT;
template <>
struct CT<float> {
  using C = float2;
};
template <>
struct CT<double> {
  using C = double2;
  using Tw = Twiddles32d;
  using U = unsigned long long;
};

__device__ __forceinline__ void sincos_r(float x, float* s, float* c) { sincos_cw(x, s, c); }

__device__ __forceinline__ void sincos_r(double x, double* s, double* c) { sincos(x, s, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float hypot_r(float a, float b) { return hypotf(a, b); }
__device__ __forceinline__ double hypot_r(double a, double b) { return hypot(a, b); }
__device__ __forceinline__ float atan2_r(float y, float x) { return atan2f(y, x); }
__device__ __forceinline__ double atan2_r(double y, double x) { return atan2(y, x); }
__device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }

// ============================================================= binning ====
// psquare_weighting lookup (native_stage2.rs:1674-1682)
template <typename R>
__device__ __forceinline__ R psquare_weight(const BinArgs& a, const R coh) {
  const double v = __dmul_rn(static_cast<double>(coh), 1000.0);
  double r = v >= 0.0 ? floor(__dadd_rn(v, 0.5)) : ceil(__dsub_rn(v, 0.5));
  r = fmin(fmax(r, 0.0), static_cast<double>(a.lut_len - 1));
  const int ix = isnan(r) ? 0 : static_cast<int>(r);
  const double t = 1.0 - a.lut[ix];
  return static_cast<R>(t * t);
}

// One warp-task of the binning: cell `task / nchunk`, interferograms
// 32 * (task % nchunk) + lane.
template <typename R, int MODE, bool ROWINV>
__device__ __forceinline__ void bin_task_t(const BinArgs& a, const int64_t task, const int lane) {
  using C = typename CT<R>::C;
  const float2* __restrict__ ph = static_cast<const float2*>(a.ph_nm);
  const R* __restrict__ K = static_cast<const R*>(a.K);
  const R* __restrict__ W = static_cast<const R*>(a.w);
  C* __restrict__ grid = static_cast<C*>(a.grid);
  const float* __restrict__ bp = a.bp;
  const int64_t M = a.M;
  {
    const int64_t cell = task / a.nchunk;
    const int chunk = static_cast<int>(task - cell * a.nchunk);
    const int c = chunk * 32 + lane;
    const bool active = c < a.M;
    const int s0 = a.cell_start[cell], s1 = a.cell_start[cell + 1];
    R ax = R(0), ay = R(0);
    // rows are taken eight at a time with every load issued before the
    // arithmetic; the sum itself stays sequential in row order
    for (int sb = s0; sb < s1; sb += 8) {
      R wv[8], kv[8], bv[8];
      float2 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int s = sb + i;
        wv[i] = R(0);
        kv[i] = R(0);
        bv[i] = R(0);
        v[i] = make_float2(0.f, 0.f);
        if (s < s1) {
          wv[i] = MODE == 3 ? R(1) : W[s];
          if (MODE != 3) kv[i] = K[s];
          if (active) {
            v[i] = ph[static_cast<int64_t>(s) * M + c];
            if (MODE != 3)
              bv[i] = ROWINV ? static_cast<R>(bp[c]) : static_cast<R>(bp[static_cast<int64_t>(s) * M + c]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int s = sb + i;
        if (s >= s1) break;
        if (!active) continue;
        if (MODE == 3) {
          // accumulate_grid alone: ph_nm holds ph_weight, no ramp and no weight
          ax = add_rn(ax, static_cast<R>(v[i].x));
          ay = add_rn(ay, static_cast<R>(v[i].y));
        } else {
          const R phs = -(bv[i] * kv[i]);
          R sn, cs;
          sincos_r(phs, &sn, &cs);
          const C r = cmul_rn(mk(static_cast<R>(v[i].x), static_cast<R>(v[i].y)), mk(cs, sn));
          ax = add_rn(ax, mul_rn(r.x, wv[i]));
          ay = add_rn(ay, mul_rn(r.y, wv[i]));
        }
      }
    }
    if (c < a.Mp) grid[cell * a.Mp + c] = active ? mk(ax, ay) : mk(R(0), R(0));
  }
}

// What an iteration needs before its binning, as one elementwise pass: K[1] <-
// K[0] (the K this iteration bins with; topofit rewrites K[0] in place), the
// statistics cleared and, from the second iteration on with P-square weighting,
// the weights of every row from its previous coherence and the table of the
// last update (the lookup once per row, not by each lane of each interferogram
// chunk inside the binning). One launch in the place of three memsets, a copy
// and a weights kernel: an iteration of a 20,000 PS x 20 patch is launch-bound
// (11 nodes -> 6 with the loop condition set by k_finalize).
template <typename R>
__global__ void __launch_bounds__(256) k_iter_begin(BeginArgs a) {
  const R* __restrict__ K0 = static_cast<const R*>(a.bin.K);
  R* __restrict__ K1 = static_cast<R*>(a.K1);
  R* __restrict__ W = static_cast<R*>(a.bin.w);
  const R* __restrict__ coh = static_cast<const R*>(a.bin.coh);
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = t0; i < a.n_partial; i += stride) a.rms_partial[i] = 0.0;
  if (t0 < kCohBins) a.hist[t0] = 0;
  if (t0 == 0) *a.n_invalid = 0;
  for (int64_t s = t0; s < a.N; s += stride) {
    K1[s] = K0[s];
    if (a.weights) W[s] = psquare_weight<R>(a.bin, coh[s]);
  }
}

cudaError_t launch_iter_begin(const BeginArgs& a, bool fp64, int sm_count, cudaStream_t st) {
  const int64_t blocks =
      std::max<int64_t>(1, std::min<int64_t>((a.N + 255) / 256, static_cast<int64_t>(sm_count) * 16));
  if (fp64)
    k_iter_begin<double><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  else
    k_iter_begin<float><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  return cudaGetLastError();
}

// The weighting mode and the row invariance of bperp are compile-time in the
// task body (no per-element branches on them).
template <typename R>
__device__ __forceinline__ void bin_task(const BinArgs& a, const int64_t task, const int lane) {
  if (a.mode == 3)
    bin_task_t<R, 3, false>(a, task, lane);
  else
    a.bp_row_inv ? bin_task_t<R, 0, true>(a, task, lane) : bin_task_t<R, 0, false>(a, task, lane);
}

// FP32: held to 64 registers so four blocks of eight warps reside per SM
// (three at its natural 76): more rows in flight against the HBM latency
// (0.281 -> 0.256 ms at 500,000 PS x 150 ifg, the same bits).
template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 1) k_bin(BinArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t ntask = a.G * a.nchunk;
  for (int64_t task = gw; task < ntask; task += nw) bin_task<R>(a, task, lane);
}

cudaError_t launch_bin(const BinArgs& a, bool fp64, int sm_count, cudaStream_t st) {
  const int64_t warps = a.G * a.nchunk;
  int64_t blocks = (warps + 7) / 8;
  // 16 blocks per SM (registers allow about three resident), or the launch shape's cap
  const int64_t cap = static_cast<int64_t>(sm_count) * (a.blocks_per_sm > 0 ? a.blocks_per_sm : 16);
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  if (fp64)
    k_bin<double><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  else
    k_bin<float><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  return cudaGetLastError();
}

// ================================================================== CLAP ==
// One warp's 32x32 working set (33-column rows avoid bank conflicts along
// columns). PAD staggers consecutive tiles: 8 floats for 4 tiles per block, 4
// for 8, so the block's interleaved loads (all tiles' ifgs of one cell at once)
// hit distinct banks.
template <typename R, int PAD>
struct ClapTileT {
  R re[32][33];
  R im[32][33];
  R hs[32][33];
  R pad[PAD];
};
template <typename R>
using ClapTile = ClapTileT<R, 8>;

// Row stride of the pyramid-weight table in shared memory: lane l reads row l,
// so rows 33 words apart put the 32 lanes on 32 different banks.
constexpr int kWtStride = 33;

// warps per CLAP block and the matching tile stagger
template <int NW>
struct ClapShape;
template <>
struct ClapShape<4> {
  static constexpr int kPad = 8;
};
__device__ __forceinline__ unsigned long long to_bits(double v) {
  return static_cast<unsigned long long>(__double_as_longlong(v));
}
__device__ __forceinline__ double from_bits(unsigned long long u) {
  return __longlong_as_double(static_cast<long long>(u));
}
__device__ __forceinline__ unsigned long long warp_min_u(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ unsigned long long warp_max_u(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// Median of the 1,024 non-negative values held 32 per lane (median(),
// native_stage2.rs:1173-1184: mean of the 512th and 513th smallest), exact.
// Bisection on the IEEE bit pattern (which orders non-negative floats like
// their values) narrows a bracket [lo, hi] holding the 512th smallest until it
// holds at most 32 of the values; those are copied to `scratch` (32 slots of
// the warp's shared memory) and ranked among themselves. v0, v1 = the 512th
// and 513th smallest.
template <typename R>
__device__ __forceinline__ void warp_median_pair(const R (&o)[32], R* scratch, R& v0, R& v1) {
  using U = typename CT<R>::U;
  const int lane = threadIdx.x & 31;
  U lo = to_bits(o[0]), hi = lo;
#pragma unroll
  for (int i = 1; i < 32; ++i) {
    const U u = to_bits(o[i]);
    lo = min(lo, u);
    hi = max(hi, u);
  }
  lo = warp_min_u(lo);
  hi = warp_max_u(hi);
  int cnt_lo = 0, cnt_hi = 1024;  // values below lo, values up to hi
  while (lo < hi && cnt_hi - cnt_lo > 32) {
    const U mid = lo + ((hi - lo) >> 1);
    unsigned cnt = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) cnt += (to_bits(o[i]) <= mid) ? 1u : 0u;
    cnt = __reduce_add_sync(kFull, cnt);
    if (cnt >= 512u) {
      hi = mid;
      cnt_hi = static_cast<int>(cnt);
    } else {
      lo = mid + 1;
      cnt_lo = static_cast<int>(cnt);
    }
  }
  const int r0 = 511 - cnt_lo;  // rank of the 512th smallest inside the bracket
  if (lo == hi) {
    v0 = from_bits(lo);
    if (cnt_hi >= 513) {
      v1 = v0;
    } else {
      U nxt = ~U(0);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const U u = to_bits(o[i]);
        if (u > hi) nxt = min(nxt, u);
      }
      v1 = from_bits(warp_min_u(nxt));
    }
    return;
  }
  // copy the bracket's values to scratch (exclusive prefix over lanes)
  int mine = 0;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const U u = to_bits(o[i]);
    mine += (u >= lo && u <= hi) ? 1 : 0;
  }
  int incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += t;
  }
  int off = incl - mine;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const U u = to_bits(o[i]);
    if (u >= lo && u <= hi) scratch[off++] = o[i];
  }
  __syncwarp();
  const int nb = cnt_hi - cnt_lo;
  const R x = lane < nb ? scratch[lane] : R(0);
  int rank = 0;
  for (int j = 0; j < nb; ++j) {
    const R y = scratch[j];
    rank += (y < x || (y == x && j < lane)) ? 1 : 0;
  }
  const unsigned m0 = __ballot_sync(kFull, lane < nb && rank == r0);
  v0 = __shfl_sync(kFull, x, __ffs(m0) - 1);
  if (r0 + 1 < nb) {
    const unsigned m1 = __ballot_sync(kFull, lane < nb && rank == r0 + 1);
    v1 = __shfl_sync(kFull, x, __ffs(m1) - 1);
  } else {
    U nxt = ~U(0);
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const U u = to_bits(o[i]);
      if (u > hi) nxt = min(nxt, u);
    }
    v1 = from_bits(warp_min_u(nxt));
  }
  __syncwarp();
}

template <typename R>
__device__ __forceinline__ R warp_median1024(const R (&o)[32], R* scratch) {
  R v0, v1;
  warp_median_pair<R>(o, scratch, v0, v1);
  return (v0 + v1) * R(0.5);
}

template <typename R>
__device__ __forceinline__ R warp_median1024_pair(const R (&o)[32], R* scratch, R& v0_out, R& v1_out) {
  warp_median_pair<R>(o, scratch, v0_out, v1_out);
  return (v0_out + v1_out) * R(0.5);
}

// One 32-point FFT per lane over a row (rows = true, lane = row) or a column
// (lane = column) of the tile, in place. The direction is a template parameter
// (every shared-memory access then has one address form); not inlined: the
// window code calls it four times and two copies keep the kernel inside the
// instruction cache. Radix-2 decimation in time (textbook Cooley-Tukey).
// tw holds e^{-2 pi i k/32} (forward) or its conjugate (inverse, no scaling: the
// 1/1024 is folded into the overlap-add weight, like rustfft's unnormalised inverse
// followed by inv_scale in the reference), k < 16.
template <typename R, bool rows, int NZ = 32>
__device__ __noinline__ void fft_pass_t(R (*re)[33], R (*im)[33], const typename CT<R>::C* tw, const int lane) {
  using C = typename CT<R>::C;
  C x[32];
  // entries NZ..31 of the row / column are zero (the window's padding) and are
  // not read
#pragma unroll
  for (int k = 0; k < 32; ++k)
    x[k] = k >= NZ ? mk(R(0), R(0)) : (rows ? mk(re[lane][k], im[lane][k]) : mk(re[k][lane], im[k][lane]));
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int r = ((i & 1) << 4) | ((i & 2) << 2) | (i & 4) | ((i & 8) >> 2) | ((i & 16) >> 4);
    if (r > i) {
      C t = x[i];
      x[i] = x[r];
      x[r] = t;
    }
  }
#pragma unroll
  for (int half = 1; half < 32; half <<= 1) {
    const int step = 16 / half;
#pragma unroll
    for (int s = 0; s < 32; s += 2 * half) {
#pragma unroll
      for (int k = 0; k < half; ++k) {
        const int ti = k * step;
        const C u = x[s + k];
        const C v = x[s + k + half];
        const C t = ti == 0 ? v : cmul(v, tw[ti]);
        x[s + k] = mk(u.x + t.x, u.y + t.y);
        x[s + k + half] = mk(u.x - t.x, u.y - t.y);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    if (rows) {
      re[lane][k] = x[k].x;
      im[lane][k] = x[k].y;
    } else {
      re[k][lane] = x[k].x;
      im[k][lane] = x[k].y;
    }
  }
}

template <typename R>
__device__ __forceinline__ void fft_pass(R (*re)[33], R (*im)[33], const typename CT<R>::C* tw, const int lane,
                                         const bool rows) {
  if (rows)
    fft_pass_t<R, true>(re, im, tw, lane);
  else
    fft_pass_t<R, false>(re, im, tw, lane);
}

// One window of one interferogram, computed by one warp in its tile.
// On entry the tile holds the 24x24 window zero-padded to 32x32; on exit rows
// and columns < n_win hold the filtered values times the pyramid weight / 1024.
template <typename R, int NWIN, typename Tile>
__device__ __forceinline__ void clap_window_warp(Tile& T, const int lane, const ClapArgs& a,
                                                 const typename CT<R>::C* twf, const typename CT<R>::C* twi,
                                                 const R* lp, const R* wt, const R (&g7)[7], const int rs,
                                                 const int cs) {
  // forward FFT along rows (rows >= n_win are zero and stay zero), then columns
  if constexpr (NWIN > 0) {
    // a compile-time window: the padding is zero by construction, never stored
    if (lane < NWIN) fft_pass_t<R, true, NWIN>(T.re, T.im, twf, lane);
    __syncwarp();
    fft_pass_t<R, false, NWIN>(T.re, T.im, twf, lane);
  } else {
    if (lane < a.n_win) fft_pass<R>(T.re, T.im, twf, lane, true);
    __syncwarp();
    fft_pass<R>(T.re, T.im, twf, lane, false);
  }
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const R xr = T.re[k][lane], xi = T.im[k][lane];
    T.hs[k][lane] = sqrt(xr * xr + xi * xi);
  }
  __syncwarp();
  // 7x7 separable Gaussian 'same' convolution of fftshift(|H|), then
  // ifftshift (native_stage2.rs:1097-1166). In unshifted coordinates this is a
  // circular convolution cut at the Nyquist seam: neighbour k+d is used iff
  // 0 <= ((k+16) mod 32) + d < 32.
  R t[32];
  const int sj = (lane + 16) & 31;
  // this lane's taps: zero where the neighbour lies across the seam (adding
  // x * 0 leaves the sum unchanged, so this equals skipping the tap)
  R gl7[7];
#pragma unroll
  for (int d = -3; d <= 3; ++d) gl7[d + 3] = (sj + d >= 0 && sj + d < 32) ? g7[d + 3] : R(0);
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    R acc = R(0);
#pragma unroll
    for (int d = -3; d <= 3; ++d) acc += T.hs[k][(lane + d) & 31] * gl7[d + 3];
    t[k] = acc;
  }
  R o[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const int sk = (k + 16) & 31;
    R acc = R(0);
#pragma unroll
    for (int d = -3; d <= 3; ++d) {
      if (sk + d >= 0 && sk + d < 32) acc += t[(k + d) & 31] * g7[d + 3];
    }
    o[k] = acc;
  }
  const R med = warp_median1024<R>(o, &T.hs[0][0]);
  // H <- max((H/med)^alpha - 1, 0); spectrum *= H*beta + low_pass
  const R beta = static_cast<R>(a.beta);
  const R alpha = static_cast<R>(a.alpha);
  const R inv_med = med != R(0) ? R(1) / med : R(1);
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    R v = o[k] * inv_med;
    v = a.alpha_is_one ? v - R(1) : pow(v, alpha) - R(1);
    if (v < R(0)) v = R(0);
    const R gk = v * beta + lp[k * 32 + lane];
    T.re[k][lane] *= gk;
    T.im[k][lane] *= gk;
  }
  // inverse FFT along columns, then rows; keep the n_win x n_win corner, weighted
  fft_pass<R>(T.re, T.im, twi, lane, false);
  __syncwarp();
  const int nwv = NWIN > 0 ? NWIN : a.n_win;
  if (lane < nwv) {
    fft_pass<R>(T.re, T.im, twi, lane, true);
    const bool row_zero = lane < rs;
    for (int l = 0; l < nwv; ++l) {
      const R wv = (row_zero || l < cs) ? R(0) : wt[(lane - rs) * kWtStride + (l - cs)];
      T.re[lane][l] *= wv;
      T.im[lane][l] *= wv;
    }
  }
  __syncwarp();
}

// Per-patch constants of the CLAP blocks: the low-pass filter and the
// pyramid weights (the twiddles and smoothing taps are the same for every patch).
template <typename R>
__device__ __forceinline__ void clap_consts(const ClapArgs& a, R* lp, R* wt) {
  const int nw2 = a.n_win * a.n_win;
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) lp[i] = static_cast<R>(a.low_pass[i]);
  for (int i = threadIdx.x; i < nw2; i += blockDim.x)
    wt[(i / a.n_win) * kWtStride + i % a.n_win] = static_cast<R>(a.wscaled[i]);
}

// Window loads and stores of a CLAP block: NW interferograms of one window,
// pixel (li, lj) of interferogram NW*g + q in tiles[q]. FP32 moves two
// interferograms (16 bytes) per access; each thread issues U accesses before
// it touches shared memory. Pixel -> (row, column) uses pix * inv_nw >> 16
// (inv_nw = ceil(65536 / nw)), exact for pix < 1024 and nw <= 32.
template <typename R>
struct ClapIo;
template <>
struct ClapIo<double> {
  static constexpr int kPer = 1;
  static constexpr int kU = 4;
};

// Interferogram c (columns >= M read as zero and are not dereferenced).
__device__ __forceinline__ void clap_fetch(const double2* p, const int c, const int M, double (&v)[2]) {
  const double2 q = c < M ? *p : make_double2(0.0, 0.0);
  v[0] = q.x;
  v[1] = q.y;
}

template <typename R, int NW, typename Tile>
__device__ __forceinline__ void clap_load_tiles(const ClapArgs& a, Tile* tiles, const typename CT<R>::C* grid,
                                                const int i1, const int j1, const int g, const int nw, const int nw2,
                                                const uint32_t inv_nw, const int tid) {
  constexpr int NT = 32 * NW, PER = ClapIo<R>::kPer, U = ClapIo<R>::kU, NQ = NW / PER;
  const int n_items = nw2 * NQ;
  for (int b0 = 0; b0 < n_items; b0 += NT * U) {
    R v[U][2 * PER];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int idx = b0 + u * NT + tid;
#pragma unroll
      for (int e = 0; e < 2 * PER; ++e) v[u][e] = R(0);
      if (idx < n_items) {
        const int pix = idx / NQ, q0 = (idx % NQ) * PER;
        const int li = static_cast<int>((static_cast<uint32_t>(pix) * inv_nw) >> 16), lj = pix - li * nw;
        const int c = NW * g + q0;
        clap_fetch(grid + (static_cast<int64_t>(i1 + li) * a.n_j + (j1 + lj)) * a.Mp + c, c, a.M, v[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int idx = b0 + u * NT + tid;
      if (idx < n_items) {
        const int pix = idx / NQ, q0 = (idx % NQ) * PER;
        const int li = static_cast<int>((static_cast<uint32_t>(pix) * inv_nw) >> 16), lj = pix - li * nw;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          R x = v[u][2 * e], y = v[u][2 * e + 1];
          if (isnan(x) || isnan(y)) x = y = R(0);  // NaN -> 0 (clap_filter_one_ifg)
          tiles[q0 + e].re[li][lj] = x;
          tiles[q0 + e].im[li][lj] = y;
        }
      }
    }
  }
}

template <typename R, int NW, typename Tile>
__device__ __forceinline__ void clap_store_tiles(const ClapArgs& a, const Tile* tiles, typename CT<R>::C* out,
                                                 const int64_t wi, const int g, const int nw, const int nw2,
                                                 const uint32_t inv_nw, const int tid) {
  constexpr int NT = 32 * NW, PER = ClapIo<R>::kPer, NQ = NW / PER;
  const int n_items = nw2 * NQ;
  for (int idx = tid; idx < n_items; idx += NT) {
    const int pix = idx / NQ, q0 = (idx % NQ) * PER;
    const int li = static_cast<int>((static_cast<uint32_t>(pix) * inv_nw) >> 16), lj = pix - li * nw;
    const int c = NW * g + q0;
    if (c >= a.Mp) continue;
    typename CT<R>::C* dst = out + (wi * nw2 + pix) * a.Mp + c;
    *dst = mk(tiles[q0].re[li][lj], tiles[q0].im[li][lj]);
  }
}

// Interferogram groups of a CLAP unit (window or window block): a task is
// (unit, group), group g holding interferograms NW * g .. NW * g + NW - 1.
template <typename R, int NW>
__device__ __forceinline__ int clap_groups(const ClapArgs& a) {
  return (a.Mp + NW - 1) / NW;
}

// Window (ix1, ix2) of interferograms NW * g + warp through the block's
// tiles: clap_windows' corner (native_stage2.rs:957-995) returned in i1, j1;
// on exit the tiles hold the weighted filtered window (rows, columns < nw).
template <typename R, int NW, int NWIN = 0>
__device__ __forceinline__ void clap_compute_window(const ClapArgs& a, const int ix1, const int ix2, const int g,
                                                    ClapTileT<R, ClapShape<NW>::kPad>* tiles,
                                                    const typename CT<R>::C* twf, const typename CT<R>::C* twi,
                                                    const R* lp, const R* wt, const R (&g7)[7], int& i1, int& j1) {
  using C = typename CT<R>::C;
  constexpr int NT = 32 * NW;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  const int n_inc = nw / 4 > 1 ? nw / 4 : 1;
  const C* __restrict__ grid = static_cast<const C*>(a.grid);
  auto& T = tiles[warp];
  i1 = ix1 * n_inc;
  int rs = 0;
  if (i1 + nw > a.n_i) {
    rs = i1 + nw - a.n_i;
    i1 = a.n_i - nw;
  }
  j1 = ix2 * n_inc;
  int cs = 0;
  if (j1 + nw > a.n_j) {
    cs = j1 + nw - a.n_j;
    j1 = a.n_j - nw;
  }
  __syncthreads();
  // zero the padding of the tiles (none for a 32-pixel window)
  if (NWIN == 0 && nw < 32) {
    for (int idx = tid; idx < NW * 32 * 32; idx += NT) {
      const int q = idx >> 10, e = idx & 1023, r = e >> 5, cc = e & 31;
      if (r >= nw || cc >= nw) {
        tiles[q].re[r][cc] = R(0);
        tiles[q].im[r][cc] = R(0);
      }
    }
  }
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  clap_load_tiles<R, NW>(a, tiles, grid, i1, j1, g, nw, nw2, inv_nw, tid);
  __syncthreads();
  if (NW * g + warp < a.M) clap_window_warp<R, NWIN>(T, lane, a, twf, twi, lp, wt, g7, rs, cs);
  __syncthreads();
}

// One block-task of the window-stack form: window a.w_lo + task / ngroups; the
// weighted window goes to win_out for the overlap-add pass.
template <typename R, int NW, int NWIN = 0>
__device__ __forceinline__ void clap_task(const ClapArgs& a, const int64_t task,
                                          ClapTileT<R, ClapShape<NW>::kPad>* tiles, const typename CT<R>::C* twf,
                                          const typename CT<R>::C* twi, const R* lp, const R* wt, const R (&g7)[7]) {
  const int ngroups = clap_groups<R, NW>(a);
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  const int64_t wi = a.w_lo + task / ngroups;
  const int g = static_cast<int>(task - (wi - a.w_lo) * ngroups);
  const int ix1 = static_cast<int>(wi / a.nwj), ix2 = static_cast<int>(wi - static_cast<int64_t>(ix1) * a.nwj);
  int i1, j1;
  clap_compute_window<R, NW, NWIN>(a, ix1, ix2, g, tiles, twf, twi, lp, wt, g7, i1, j1);
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  clap_store_tiles<R, NW>(a, tiles, static_cast<typename CT<R>::C*>(a.win_out), wi, g, nw, nw2, inv_nw,
                          threadIdx.x);
}

// ---- overlap-add fused into the window pass (window blocks) -------------------
// The windows are taken in blocks of 4 x 4 (window rows 4 bi .. 4 bi + 3,
// columns 4 bj .. 4 bj + 3). A block's windows cover a box of at most
// clap_box(n_win) = 3 n_inc + n_win cells a side from the corner of its first
// window; one block-task runs the block's windows in order (ix1, then ix2) for
// NW interferograms and adds each weighted window into the block's FP64
// partial sum of the box (part: [block][box row][box column][Mp] of complex
// FP64; the first window of the block that covers a cell stores instead of
// adding), so a cell's partial is the reference's ordered sum
// (native_stage2.rs:1166-1184) over the block's windows. The combine pass
// adds a cell's block partials (2 x 2 at most for 24-cell windows) in block
// order and rounds once. The window stack of the two-pass form (1.1 GB for a
// 256 x 256 x 150 grid) is never written; the partials are 2.7x the grid and a
// block's box stays in L2 while its windows run.
// Add (or store, for a cell no earlier window of the block covered) the
// weighted window in the tiles to the block partial. Box corner (r0, c0); pi1 /
// pj1 the corner row / column of the block's previous window row / column
// (rows < pi1 + nw were covered already), or a value that marks none. One item
// per (pixel, interferogram): NW consecutive threads write one cell's NW
// interferograms, 16 * NW contiguous bytes; each thread issues the partial
// loads of kAccBatch items before any add, so their L2 round trips overlap.
constexpr int kAccBatch = 6;
template <typename R, int NW, typename Tile>
__device__ __forceinline__ void clap_accum_tiles(const ClapArgs& a, const Tile* tiles, double2* __restrict__ part,
                                                 const int64_t blk, const int box, const int i1, const int j1,
                                                 const int r0, const int c0, const int pi1, const int pj1,
                                                 const int g, const int nw, const int nw2, const uint32_t inv_nw,
                                                 const int tid) {
  constexpr int NT = 32 * NW;
  const int n_items = nw2 * NW;
  for (int b0 = tid; b0 < n_items; b0 += NT * kAccBatch) {
    double2 old[kAccBatch];
    int64_t off[kAccBatch];
    int li[kAccBatch], lj[kAccBatch], qq[kAccBatch];
    bool live[kAccBatch], first[kAccBatch];
#pragma unroll
    for (int u = 0; u < kAccBatch; ++u) {
      const int idx = b0 + u * NT;
      const int pix = idx / NW, q = idx - (idx / NW) * NW;
      const int c = NW * g + q;
      live[u] = idx < n_items && c < a.M;
      li[u] = static_cast<int>((static_cast<uint32_t>(pix) * inv_nw) >> 16);
      lj[u] = pix - li[u] * nw;
      qq[u] = q;
      const int ai = i1 + li[u], aj = j1 + lj[u];
      first[u] = ai >= pi1 + nw && aj >= pj1 + nw;
      off[u] = ((blk * box + (ai - r0)) * box + (aj - c0)) * a.Mp + c;
      old[u] = make_double2(0.0, 0.0);
      if (live[u] && !first[u]) old[u] = part[off[u]];
    }
#pragma unroll
    for (int u = 0; u < kAccBatch; ++u) {
      if (!live[u]) continue;
      const double vx = static_cast<double>(tiles[qq[u]].re[li[u]][lj[u]]);
      const double vy = static_cast<double>(tiles[qq[u]].im[li[u]][lj[u]]);
      part[off[u]] = first[u] ? make_double2(vx, vy) : make_double2(__dadd_rn(old[u].x, vx), __dadd_rn(old[u].y, vy));
    }
  }
}

// One block-task of the fused form: window block a.w_lo + task / ngroups.
template <typename R, int NW, int NWIN = 0>
__device__ __forceinline__ void clap_block_task(const ClapArgs& a, const int64_t task,
                                                ClapTileT<R, ClapShape<NW>::kPad>* tiles,
                                                const typename CT<R>::C* twf, const typename CT<R>::C* twi,
                                                const R* lp, const R* wt, const R (&g7)[7]) {
  const int ngroups = clap_groups<R, NW>(a);
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  const int n_inc = nw / 4 > 1 ? nw / 4 : 1;
  const int box = clap_box(nw);
  const int nbj = clap_block_rows(a.nwj);
  const int64_t blk = a.w_lo + task / ngroups;
  const int g = static_cast<int>(task - (blk - a.w_lo) * ngroups);
  const int bi = static_cast<int>(blk / nbj), bj = static_cast<int>(blk - static_cast<int64_t>(bi) * nbj);
  const int ixa = kClapBlockWin * bi, ixb = min(ixa + kClapBlockWin, a.nwi);
  const int jxa = kClapBlockWin * bj, jxb = min(jxa + kClapBlockWin, a.nwj);
  const int r0 = min(ixa * n_inc, a.n_i - nw), c0 = min(jxa * n_inc, a.n_j - nw);
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  double2* part = static_cast<double2*>(a.part);
  constexpr int kNone = -(1 << 20);
  for (int ix1 = ixa; ix1 < ixb; ++ix1) {
    const int pi1 = ix1 > ixa ? min((ix1 - 1) * n_inc, a.n_i - nw) : kNone;
    for (int ix2 = jxa; ix2 < jxb; ++ix2) {
      const int pj1 = ix2 > jxa ? min((ix2 - 1) * n_inc, a.n_j - nw) : kNone;
      int i1, j1;
      clap_compute_window<R, NW, NWIN>(a, ix1, ix2, g, tiles, twf, twi, lp, wt, g7, i1, j1);
      clap_accum_tiles<R, NW>(a, tiles, part, blk, box, i1, j1, r0, c0, pi1, pj1, g, nw, nw2, inv_nw,
                              threadIdx.x);
    }
  }
}

// shared-memory carve-up of a CLAP block: NW tiles, low-pass, weights, twiddles
template <typename R, int NW>
struct ClapSmem {
  ClapTileT<R, ClapShape<NW>::kPad>* tiles;
  R* lp;
  R* wt;
  typename CT<R>::C* twf;
  typename CT<R>::C* twi;
};

template <typename R, int NW>
__device__ __forceinline__ ClapSmem<R, NW> clap_smem(unsigned char* raw, const typename CT<R>::Tw& tw) {
  ClapSmem<R, NW> m;
  m.tiles = reinterpret_cast<ClapTileT<R, ClapShape<NW>::kPad>*>(raw);
  m.lp = reinterpret_cast<R*>(m.tiles + NW);
  m.wt = m.lp + 1024;
  m.twf = reinterpret_cast<typename CT<R>::C*>(m.wt + 32 * kWtStride);
  m.twi = m.twf + 16;
  if (threadIdx.x < 16) {
    m.twf[threadIdx.x] = tw.w[threadIdx.x];
    m.twi[threadIdx.x] = mk(tw.w[threadIdx.x].x, -tw.w[threadIdx.x].y);
  }
  return m;
}

// FUSED: window blocks into the partials; otherwise windows into the window stack.
template <typename R, int NW, int NWIN, bool FUSED>
__global__ void __launch_bounds__(32 * NW, 1)
    k_clap(ClapArgs a, typename CT<R>::Tw tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ClapSmem<R, NW> m = clap_smem<R, NW>(smem_raw, tw);
  clap_consts<R>(a, m.lp, m.wt);
  R g7[7];
#pragma unroll
  for (int i = 0; i < 7; ++i) g7[i] = static_cast<R>(a.g7[i]);
  // units: window blocks (fused) or windows (window stack)
  const int64_t nunit = a.w_n > 0 ? a.w_n
                        : FUSED ? static_cast<int64_t>(clap_block_rows(a.nwi)) * clap_block_rows(a.nwj)
                                : static_cast<int64_t>(a.nwi) * a.nwj;
  const int64_t ntask = nunit * clap_groups<R, NW>(a);
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    if constexpr (FUSED)
      clap_block_task<R, NW, NWIN>(a, task, m.tiles, m.twf, m.twi, m.lp, m.wt, g7);
    else
      clap_task<R, NW, NWIN>(a, task, m.tiles, m.twf, m.twi, m.lp, m.wt, g7);
  }
}

template <typename R, int NW>
static size_t clap_smem_bytes() {
  return NW * sizeof(ClapTileT<R, ClapShape<NW>::kPad>) + (1024 + 32 * kWtStride) * sizeof(R) + 32 * 2 * sizeof(R);
}

template <typename R, int NW, int NWIN>
static cudaError_t launch_clap_nwin(const ClapArgs& a, const typename CT<R>::Tw& tw, int sm_count, cudaStream_t st) {
  if (a.nwi <= 0 || a.nwj <= 0) return cudaSuccess;
  const int64_t nunit = a.w_n > 0 ? a.w_n
                        : a.part ? static_cast<int64_t>(clap_block_rows(a.nwi)) * clap_block_rows(a.nwj)
                                 : static_cast<int64_t>(a.nwi) * a.nwj;
  const int64_t ntask = nunit * ((a.Mp + NW - 1) / NW);
  if (ntask <= 0) return cudaSuccess;
  const size_t sm = clap_smem_bytes<R, NW>();
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  if (a.part)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clap<R, NW, NWIN, true>, 32 * NW, sm);
  else
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clap<R, NW, NWIN, false>, 32 * NW, sm);
  if (e != cudaSuccess) return e;
  if (a.blocks_per_sm > 0 && a.blocks_per_sm < per_sm) per_sm = a.blocks_per_sm;
  const int64_t blocks = std::min<int64_t>(ntask, static_cast<int64_t>(sm_count) * (per_sm > 0 ? per_sm : 1));
  if (a.part)
    k_clap<R, NW, NWIN, true><<<static_cast<unsigned>(blocks), 32 * NW, sm, st>>>(a, tw);
  else
    k_clap<R, NW, NWIN, false><<<static_cast<unsigned>(blocks), 32 * NW, sm, st>>>(a, tw);
  return cudaGetLastError();
}

// the 24-pixel window (clap_win 32 x 0.75) as a compile-time shape, others at run time
template <typename R, int NW>
static cudaError_t launch_clap_nw(const ClapArgs& a, const typename CT<R>::Tw& tw, int sm_count, cudaStream_t st) {
  return a.n_win == 24 ? launch_clap_nwin<R, NW, 24>(a, tw, sm_count, st) : launch_clap_nwin<R, NW, 0>(a, tw, sm_count, st);
}

// FP32 is in clap_f32.cu. Every window's arithmetic is the same whatever the shape.
cudaError_t launch_clap(const ClapArgs& a, bool fp64, const Twiddles32d& td, int sm_count, cudaStream_t st) {
  return fp64 ? launch_clap_nw<double, 4>(a, td, sm_count, st) : launch_clap_f32(a, sm_count, st);
}

// Overlap-add as a gather: cell (i, j) sums the windows that cover it, in the
// reference's raster window order, in f64 (the reference accumulates in f64).
// QUARTERS: n_win is a multiple of 4, windows n_win / 4 apart; 4 or 5 of them cover a
// cell along an axis. Other sizes have n_inc = n_win / 4 rounded down and up to 10.
template <typename R, bool QUARTERS>
__device__ __forceinline__ void overlap_elem(const OverlapArgs& a, const int64_t idx) {
  using C = typename CT<R>::C;
  const C* __restrict__ win = static_cast<const C*>(a.win_out);
  C* __restrict__ filt = static_cast<C*>(a.filt);
  const int nw = a.n_win, nw2 = nw * nw;
  {
    const int64_t cell = idx / a.Mp;
    const int c = static_cast<int>(idx - cell * a.Mp);
    const int i = static_cast<int>(cell / a.n_j), j = static_cast<int>(cell - static_cast<int64_t>(i) * a.n_j);
    double sx = 0.0, sy = 0.0;
    if (c < a.M && a.nwi > 0 && a.nwj > 0) {
      const int qi = i / a.n_inc, qj = j / a.n_inc;
      if constexpr (QUARTERS) {
        // windows q - 3 .. q cover the cell, and the last one, clamped to the edge, may
        const int a1 = max(0, qi - 3), b1 = min(a.nwi - 1, qi + 1);
        const int a2 = max(0, qj - 3), b2 = min(a.nwj - 1, qj + 1);
        // the (at most 5) candidate windows along j, their offsets and validity
        int lj5[5];
        bool ok5[5];
#pragma unroll
        for (int w = 0; w < 5; ++w) {
          const int ix2 = a2 + w;
          const int lj = j - min(ix2 * a.n_inc, a.n_j - nw);
          ok5[w] = ix2 <= b2 && lj >= 0;
          lj5[w] = lj;
        }
        for (int ix1 = a1; ix1 <= b1; ++ix1) {
          const int li = i - min(ix1 * a.n_inc, a.n_i - nw);
          if (li < 0) continue;
          // one row of covering windows: every load issued before the ordered sum
          C v[5];
#pragma unroll
          for (int w = 0; w < 5; ++w)
            v[w] = ok5[w] ? win[((static_cast<int64_t>(ix1) * a.nwj + a2 + w) * nw2 + li * nw + lj5[w]) * a.Mp + c]
                          : mk(R(0), R(0));
#pragma unroll
          for (int w = 0; w < 5; ++w)
            if (ok5[w]) {
              sx += static_cast<double>(v[w].x);
              sy += static_cast<double>(v[w].y);
            }
        }
      } else {
        // window ix starts at min(ix n_inc, n - nw): those that cover a cell are a run,
        // up to the last window (with others clamped alike) for an edge window's cells
        const int a1 = i < nw ? 0 : (i - nw) / a.n_inc + 1, b1 = i >= a.n_i - nw ? a.nwi - 1 : min(a.nwi - 1, qi);
        const int a2 = j < nw ? 0 : (j - nw) / a.n_inc + 1, b2 = j >= a.n_j - nw ? a.nwj - 1 : min(a.nwj - 1, qj);
        for (int ix1 = a1; ix1 <= b1; ++ix1) {
          const int li = i - min(ix1 * a.n_inc, a.n_i - nw);
          for (int ix2 = a2; ix2 <= b2; ++ix2) {
            const int lj = j - min(ix2 * a.n_inc, a.n_j - nw);
            const C v = win[((static_cast<int64_t>(ix1) * a.nwj + ix2) * nw2 + li * nw + lj) * a.Mp + c];
            sx += static_cast<double>(v.x);
            sy += static_cast<double>(v.y);
          }
        }
      }
    }
    C f = mk(static_cast<R>(sx), static_cast<R>(sy));
    if (a.normalize) {
      // normalize_complex_unit_magnitude (:1186-1205) once per cell instead of
      // once per PS of the cell in the topofit; the same expression, the same bits
      const R mag = hypot_r(f.x, f.y);
      if (mag != R(0)) f = mk(f.x / mag, f.y / mag);
    }
    filt[idx] = f;
  }
}

// Fused form: the cell's block partials (those whose boxes hold the cell: 2 x 2
// at most for 24-cell windows) added in block order in FP64, then rounded and
// normalised as overlap_elem does.
template <typename R>
__device__ __forceinline__ void combine_elem(const OverlapArgs& a, const int64_t idx) {
  using C = typename CT<R>::C;
  const double2* __restrict__ part = static_cast<const double2*>(a.part);
  C* __restrict__ filt = static_cast<C*>(a.filt);
  const int nw = a.n_win, box = clap_box(nw);
  const int64_t cell = idx / a.Mp;
  const int c = static_cast<int>(idx - cell * a.Mp);
  const int i = static_cast<int>(cell / a.n_j), j = static_cast<int>(cell - static_cast<int64_t>(i) * a.n_j);
  double sx = 0.0, sy = 0.0;
  if (c < a.M && a.nwi > 0 && a.nwj > 0) {
    const int nbi = clap_block_rows(a.nwi), nbj = clap_block_rows(a.nwj);
    // blocks whose boxes [corner of the first window, corner of the last + nw)
    // hold (i, j), in block order: the box corners do not decrease along an
    // axis, and no box that holds i starts before block (i - nw) / (4 n_inc) - 1
    const int bj_lo = max(0, (j - nw) / (kClapBlockWin * a.n_inc) - 1);
    for (int bi = max(0, (i - nw) / (kClapBlockWin * a.n_inc) - 1); bi < nbi; ++bi) {
      const int r0 = min(kClapBlockWin * bi * a.n_inc, a.n_i - nw);
      if (r0 > i) break;
      const int r1 = min((min(kClapBlockWin * bi + kClapBlockWin, a.nwi) - 1) * a.n_inc, a.n_i - nw) + nw;
      if (i >= r1) continue;
      for (int bj = bj_lo; bj < nbj; ++bj) {
        const int c0 = min(kClapBlockWin * bj * a.n_inc, a.n_j - nw);
        if (c0 > j) break;
        const int c1 = min((min(kClapBlockWin * bj + kClapBlockWin, a.nwj) - 1) * a.n_inc, a.n_j - nw) + nw;
        if (j >= c1) continue;
        const int64_t blk = static_cast<int64_t>(bi) * nbj + bj;
        const double2 p = part[((blk * box + (i - r0)) * box + (j - c0)) * a.Mp + c];
        sx = __dadd_rn(sx, p.x);
        sy = __dadd_rn(sy, p.y);
      }
    }
  }
  C f = mk(static_cast<R>(sx), static_cast<R>(sy));
  if (a.normalize) {
    const R mag = hypot_r(f.x, f.y);
    if (mag != R(0)) f = mk(f.x / mag, f.y / mag);
  }
  filt[idx] = f;
}

template <typename R>
__device__ __forceinline__ void overlap_any(const OverlapArgs& a, const int64_t idx) {
  if (a.part)
    combine_elem<R>(a, idx);
  else if (a.n_win % 4 == 0)
    overlap_elem<R, true>(a, idx);
  else
    overlap_elem<R, false>(a, idx);
}

template <typename R>
__global__ void __launch_bounds__(256) k_overlap(OverlapArgs a) {
  const int64_t cells = a.cell_n > 0 ? a.cell_n : static_cast<int64_t>(a.n_i) * a.n_j;
  const int64_t total = cells * a.Mp, base = a.cell_lo * a.Mp;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x)
    overlap_any<R>(a, base + idx);
}

cudaError_t launch_overlap(const OverlapArgs& a, bool fp64, cudaStream_t st) {
  const int64_t cells = a.cell_n > 0 ? a.cell_n : static_cast<int64_t>(a.n_i) * a.n_j;
  const int64_t total = cells * a.Mp;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  if (fp64)
    k_overlap<double><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  else
    k_overlap<float><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  return cudaGetLastError();
}

// Plain FP64 topofit, the comparison path; it shares only the data layout with
// the FP32 kernel. A direct sincos for every (trial, column) made it 77 % of an
// FP64 iteration. A warp takes 32 / L rows: their z and theta go to shared memory
// (lanes over columns, a row at a time); the trial sums of the rows run side by
// side (L = 8 or 16 lanes a row, lanes over columns) as phasor chains, trials +-m from one
// chain; each row's refinement is again the warp's, lanes over columns. The
// chains only rank the trials: where the best one does not lead by more than
// their rounding error, the row's trials are evaluated again by the direct sum
// (every lane its trials, columns in order), so the trial chosen is the direct
// sum's. 100,000 PS x 40 ifg x 121 trials: 1.73 -> 0.57 ms.
constexpr int kF64Warps = 2, kF64W = 8;

// Columns padded to the L lanes of a row.
template <int L>
__host__ __device__ inline int f64_mpad(int M) {
  return (M + L - 1) / L * L;
}
// Row stride in columns: an odd multiple of 8, so that the rows of a warp start in
// different banks.
template <int L>
__host__ __device__ inline int f64_stride(int M) {
  return (f64_mpad<L>(M) / 8) % 2 ? f64_mpad<L>(M) : f64_mpad<L>(M) + 8;
}
// z, rotation and phasor per column: 48 bytes; at M = 150 and 16 lanes a row 32 KB a
// block, fourteen warps an SM
template <int L>
static size_t topofit_f64_smem(int M) {
  return static_cast<size_t>(kF64Warps) * (32 / L) * f64_stride<L>(M) * 3 * sizeof(double2);
}

// Trial -> best |S|^2, its trial (the first on ties) and the largest |S|^2 among the others.
struct Top2 {
  double best, second;
  int t;
  __device__ __forceinline__ void add(double v, int tt) {
    if (v > best || (v == best && tt < t)) {
      second = best;
      best = v;
      t = tt;
    } else if (v > second) {
      second = v;
    }
  }
};

template <int L>
__global__ void __launch_bounds__(32 * kF64Warps) k_topofit_f64(TopoArgs a) {
  constexpr int PS = 32 / L;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int stride = f64_stride<L>(a.M), mpad = f64_mpad<L>(a.M);
  double2* zs0 = reinterpret_cast<double2*>(smem_raw) + static_cast<int64_t>(wib) * PS * stride * 3;
  double2* rot0 = zs0 + PS * stride;
  double2* ph0 = rot0 + PS * stride;
  __shared__ int sh_hist[kCohBins];
  __shared__ double sh_rms[kF64Warps];
  __shared__ int sh_inv[kF64Warps];
  __shared__ double sh_row[kF64Warps][PS][4];  // per row: range, largest |bp| then trial K, refined K, sums
  for (int i = tid; i < kCohBins; i += blockDim.x) sh_hist[i] = 0;
  __syncthreads();
  const float2* __restrict__ ph_nm = static_cast<const float2*>(a.ph_nm);
  const double2* __restrict__ filt = static_cast<const double2*>(a.filt);
  double* K_out = static_cast<double*>(a.K_out);
  double* C_out = static_cast<double*>(a.C_out);
  double* coh_io = static_cast<double*>(a.coh_io);
  double2* resid = static_cast<double2*>(a.residual);
  double* ph_res = static_cast<double*>(a.ph_res);
  double2* ph_patch = static_cast<double2*>(a.ph_patch);
  const int64_t M = a.M;
  const int T = 2 * a.n_half + 1;
  const double qpi = 3.14159265358979323846 / 4.0;
  double rms_acc = 0.0;
  int inv_acc = 0;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + tid) >> 5;
  const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int g = lane / L, gl = lane % L;
  for (int64_t s0 = gw * PS; s0 < a.N; s0 += nwarps * PS) {
    const int rows = a.N - s0 < PS ? static_cast<int>(a.N - s0) : PS;
    unsigned invalid_rows = 0;
    __syncwarp();
    // elementwise steps run over all elements of the rows, so that no lane idles at
    // the end of each row
    const int total = rows * a.M;
    for (int idx = lane; idx < total; idx += 32) {
      const int q = idx / a.M, c = idx - q * a.M;
      const int64_t s = s0 + q, cell = a.cell_of[s];
      double2 f = filt[cell * a.Mp + c];
      if (!a.filt_unit) {
        const double mag = hypot(f.x, f.y);
        if (mag != 0.0) f = make_double2(f.x / mag, f.y / mag);
      }
      if (ph_patch) ph_patch[s * M + c] = f;
      const float2 p = ph_nm[s * M + c];
      zs0[q * stride + c] = cmul_rn(conjd2(f), make_double2(p.x, p.y));
      rot0[q * stride + c].x = a.bp_row_inv ? static_cast<double>(a.bp[c]) : static_cast<double>(a.bp[s * M + c]);
    }
    __syncwarp();
    for (int q = 0; q < rows; ++q) {
      bool zero = false;
      double mn = INFINITY, mx = -INFINITY;
      for (int c = lane; c < a.M; c += 32) {
        const double2 v = zs0[q * stride + c];
        if (v.x == 0.0 && v.y == 0.0) zero = true;
        const double b = rot0[q * stride + c].x;
        mn = fmin(mn, b);
        mx = fmax(mx, b);
      }
      if (__any_sync(kFull, zero)) invalid_rows |= 1u << q;
      mn = warp_min(mn);
      mx = warp_max(mx);
      double range = mx - mn;
      if (range == 0.0) range = 1.0;
      if (lane == 0) {
        sh_row[wib][q][0] = range;
        sh_row[wib][q][1] = fmax(fabs(mn), fabs(mx));
      }
    }
    __syncwarp();
    for (int idx = lane; idx < rows * mpad; idx += 32) {
      const int q = idx / mpad, c = idx - q * mpad;
      const bool in = c < a.M;
      const double th = in ? (rot0[q * stride + c].x / sh_row[wib][q][0]) * qpi : 0.0;
      if (!in) zs0[q * stride + c] = make_double2(0.0, 0.0);
      double sn, cs;
      sincos(th, &sn, &cs);
      rot0[q * stride + c] = make_double2(cs, -sn);
      ph0[q * stride + c] = make_double2(cs, -sn);  // |m| = 1
    }
    __syncwarp();
    // trial chains of row s0 + g over the lane's columns gl, gl + 8, ...: with
    // w = e^{-j m theta}, z w is trial +m and z conj(w) trial -m
    Top2 top{-1.0, -1.0, a.n_half};
    double zz = 0.0, sx0 = 0.0, sy0 = 0.0;
    if (g < rows) {
      const double2* zs = zs0 + g * stride;
      for (int c = gl; c < mpad; c += L) {
        const double2 z = zs[c];
        sx0 += z.x;
        sy0 += z.y;
        zz += z.x * z.x + z.y * z.y;
      }
    }
    sx0 = group_sum<L>(sx0);
    sy0 = group_sum<L>(sy0);
    zz = group_sum<L>(zz);
    if (gl == 0) top.add(sx0 * sx0 + sy0 * sy0, a.n_half);
    for (int m0 = 1; m0 <= a.n_half; m0 += kF64W) {
      double2 A[kF64W], B[kF64W];  // (sum x w.x, sum x w.y), (sum y w.x, sum y w.y)
#pragma unroll
      for (int i = 0; i < kF64W; ++i) A[i] = B[i] = make_double2(0.0, 0.0);
      if (g < rows) {
        const double2* zs = zs0 + g * stride;
        const double2* rot = rot0 + g * stride;
        double2* ph = ph0 + g * stride;
        for (int c = gl; c < mpad; c += L) {
          const double2 z = zs[c], r = rot[c];
          double2 w = ph[c];
#pragma unroll
          for (int i = 0; i < kF64W; ++i) {
            A[i].x = fma(z.x, w.x, A[i].x);
            A[i].y = fma(z.x, w.y, A[i].y);
            B[i].x = fma(z.y, w.x, B[i].x);
            B[i].y = fma(z.y, w.y, B[i].y);
            w = make_double2(fma(w.x, r.x, -(w.y * r.y)), fma(w.x, r.y, w.y * r.x));
          }
          ph[c] = w;
        }
      }
      // slots 0..7: trials +(m0 + i); 8..15: trials -(m0 + i); halved over the
      // group's lanes until each holds two
      double2 S[2 * kF64W];
#pragma unroll
      for (int i = 0; i < kF64W; ++i) {
        S[i] = make_double2(A[i].x - B[i].y, A[i].y + B[i].x);
        S[kF64W + i] = make_double2(A[i].x + B[i].y, B[i].x - A[i].y);
      }
      int base = 0;
#pragma unroll
      for (int o = L / 2, h = kF64W; o >= 1; o >>= 1, h >>= 1) {
        const bool upper = (gl & o) != 0;
#pragma unroll
        for (int i = 0; i < kF64W; ++i) {
          if (i < h) {
            const double2 lo = S[i], hi = S[i + h];
            const double2 keep = upper ? hi : lo;
            double2 send = upper ? lo : hi;
            send.x = __shfl_xor_sync(kFull, send.x, o);
            send.y = __shfl_xor_sync(kFull, send.y, o);
            S[i] = make_double2(keep.x + send.x, keep.y + send.y);
          }
        }
        if (upper) base += h;
      }
#pragma unroll
      for (int i = 0; i < 2 * kF64W / L; ++i) {
        const int idx = base + i, m = m0 + (idx < kF64W ? idx : idx - kF64W);
        if (m <= a.n_half) top.add(S[i].x * S[i].x + S[i].y * S[i].y, idx < kF64W ? a.n_half + m : a.n_half - m);
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(kFull, top.best, o), os = __shfl_xor_sync(kFull, top.second, o);
      const int ot = __shfl_xor_sync(kFull, top.t, o);
      const bool theirs = ob > top.best || (ob == top.best && ot < top.t);
      top.second = fmax(theirs ? top.best : ob, theirs ? os : top.second);
      if (theirs) {
        top.best = ob;
        top.t = ot;
      }
    }
    // a chain's phasor is off by at most ~3e-16 a step, the direct sum's by the
    // rounding of its argument theta m (2^-53 of it), a sum by that times sum |z|,
    // its square by 2 (sum |z|)^2 times that; (sum |z|)^2 <= M sum |z|^2, and two
    // squares are compared. theta is large where the baselines lie close together
    // far from zero
    const float th_max = static_cast<float>(sh_row[wib][g < rows ? g : 0][1]) /
                         static_cast<float>(sh_row[wib][g < rows ? g : 0][0]);  // in units of pi / 4
    const double tol = (4.0e-15 * (a.n_half + 64) + 4.0e-16 * th_max * a.n_half) * a.M * zz;
    const unsigned clear = __ballot_sync(kFull, top.best - top.second > tol);
    for (int q = 0; q < rows; ++q) {
      const int64_t s = s0 + q;
      const double2* zs = zs0 + q * stride;
      double2* rot = rot0 + q * stride;
      const double range = sh_row[wib][q][0];
      int bt = __shfl_sync(kFull, top.t, q * L);
      if (!((invalid_rows >> q) & 1u) && !((clear >> (q * L)) & 1u)) {
        for (int c = lane; c < a.M; c += 32) {
          const double b = a.bp_row_inv ? static_cast<double>(a.bp[c]) : static_cast<double>(a.bp[s * M + c]);
          rot[c].x = (b / range) * qpi;
        }
        __syncwarp();
        double best = -1.0;
        bt = 0;
        for (int t = lane; t < T; t += 32) {
          const double m = static_cast<double>(t - a.n_half);
          double sx = 0.0, sy = 0.0;
          for (int c = 0; c < a.M; ++c) {
            double sn, cs;
            sincos(rot[c].x * m, &sn, &cs);
            const double2 z = zs[c];
            sx += z.x * cs + z.y * sn;
            sy += z.y * cs - z.x * sn;
          }
          const double sq = sx * sx + sy * sy;
          if (sq > best) {
            best = sq;
            bt = t;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(kFull, best, o);
          const int ot = __shfl_xor_sync(kFull, bt, o);
          if (ob > best || (ob == best && ot < bt)) {
            best = ob;
            bt = ot;
          }
        }
        __syncwarp();
      }
      if (lane == 0) sh_row[wib][q][1] = qpi / range * static_cast<double>(bt - a.n_half);
    }
    __syncwarp();
    auto bperp = [&](int64_t s, int c) {
      return a.bp_row_inv ? static_cast<double>(a.bp[c]) : static_cast<double>(a.bp[s * M + c]);
    };
    // refine_candidate (native_stage2.rs:1259-1303): elements of all rows, then each
    // row's sums (lanes over its columns)
    for (int idx = lane; idx < total; idx += 32) {
      const int q = idx / a.M, c = idx - q * a.M;
      double sn, cs;
      sincos(sh_row[wib][q][1] * bperp(s0 + q, c), &sn, &cs);
      rot0[q * stride + c] = cmul_rn(zs0[q * stride + c], make_double2(cs, -sn));
    }
    __syncwarp();
    for (int q = 0; q < rows; ++q) {
      double ox = 0.0, oy = 0.0;
      for (int c = lane; c < a.M; c += 32) {
        ox += rot0[q * stride + c].x;
        oy += rot0[q * stride + c].y;
      }
      ox = warp_sum(ox);
      oy = warp_sum(oy);
      if (lane == 0) {
        sh_row[wib][q][2] = ox;
        sh_row[wib][q][3] = oy;
      }
    }
    __syncwarp();
    for (int idx = lane; idx < total; idx += 32) {
      const int q = idx / a.M, c = idx - q * a.M;
      const double2 z = zs0[q * stride + c];
      const double wgt = hypot(z.x, z.y);
      const double2 x = cmul_rn(rot0[q * stride + c], make_double2(sh_row[wib][q][2], -sh_row[wib][q][3]));
      ph0[q * stride + c] = make_double2(wgt * bperp(s0 + q, c), wgt * atan2(x.y, x.x));
    }
    __syncwarp();
    for (int q = 0; q < rows; ++q) {
      double mopt = 0.0, dl = 0.0;
      for (int c = lane; c < a.M; c += 32) {
        const double2 x = ph0[q * stride + c];
        dl = fma(x.x, x.x, dl);
        mopt = fma(x.x, x.y, mopt);
      }
      mopt = warp_sum(mopt);
      dl = warp_sum(dl);
      if (dl == 0.0) dl = 1.0;
      if (lane == 0) sh_row[wib][q][2] = sh_row[wib][q][1] + mopt / dl;
    }
    __syncwarp();
    for (int idx = lane; idx < total; idx += 32) {
      const int q = idx / a.M, c = idx - q * a.M;
      const int64_t s = s0 + q;
      double sn, cs;
      sincos(sh_row[wib][q][2] * bperp(s, c), &sn, &cs);
      const double2 r = cmul_rn(zs0[q * stride + c], make_double2(cs, -sn));
      rot0[q * stride + c] = r;
      ph0[q * stride + c].x = hypot(r.x, r.y);
      const bool bad = (invalid_rows >> q) & 1u;
      if (resid) resid[s * M + c] = bad ? make_double2(0.0, 0.0) : r;
      if (ph_res) ph_res[s * M + c] = bad ? 0.0 : atan2(r.y, r.x);
    }
    __syncwarp();
    double mx2 = 0.0, my2 = 0.0, den2 = 0.0;  // of row s0 + lane
    for (int q = 0; q < rows; ++q) {
      double x = 0.0, y = 0.0, d = 0.0;
      for (int c = lane; c < a.M; c += 32) {
        x += rot0[q * stride + c].x;
        y += rot0[q * stride + c].y;
        d += ph0[q * stride + c].x;
      }
      x = warp_sum(x);
      y = warp_sum(y);
      d = warp_sum(d);
      if (lane == q) {
        mx2 = x;
        my2 = y;
        den2 = d;
      }
    }
    if (lane < rows) {
      const int64_t s = s0 + lane;
      const bool bad = (invalid_rows >> lane) & 1u;
      double Kv = __longlong_as_double(0x7ff8000000000000LL), Cv = 0.0, cohv = 0.0;
      if (bad) {
        inv_acc += 1;
      } else {
        if (den2 == 0.0) den2 = 1.0;
        Kv = sh_row[wib][lane][2];
        Cv = atan2(my2, mx2);
        cohv = hypot(mx2, my2) / den2;
      }
      if (a.accumulate_stats) {
        const double d = cohv - coh_io[s];
        rms_acc += d * d;
        const int b = coh_bin(cohv, a.cutoff0, a.dbin);
        if (b >= 0) atomicAdd(&sh_hist[b], 1);
      }
      K_out[s] = Kv;
      C_out[s] = Cv;
      coh_io[s] = cohv;
      if (a.nopt) a.nopt[s] = bad ? 0 : 1;
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
    double t = 0.0;
    int iv = 0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
      t += sh_rms[w];
      iv += sh_inv[w];
    }
    a.rms_partial[blockIdx.x] = t;
    if (iv) atomicAdd(a.n_invalid, iv);
  }
  for (int i = tid; i < kCohBins; i += blockDim.x)
    if (sh_hist[i]) atomicAdd(&a.hist[i], sh_hist[i]);
}

int topofit_grid_blocks(int sm_count, bool fp64) { return sm_count * 16; }

int clap_block_count(int nw_axis) { return clap_block_rows(nw_axis); }

int64_t clap_part_elems(int nwi, int nwj, int n_win, int Mp) {
  const int64_t box = clap_box(n_win);
  return std::max<int64_t>(static_cast<int64_t>(clap_block_rows(nwi)) * clap_block_rows(nwj), 1) * box * box * Mp;
}

template <int L>
static cudaError_t launch_topofit_f64(const TopoArgs& a, int grid_blocks, cudaStream_t st) {
  const int64_t per_block = kF64Warps * (32 / L);
  const int blocks = static_cast<int>(std::min<int64_t>((a.N + per_block - 1) / per_block, grid_blocks));
  const size_t sm = topofit_f64_smem<L>(a.M);
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  k_topofit_f64<L><<<blocks, 32 * kF64Warps, sm, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_topofit(const TopoArgs& a, bool fp64, int grid_blocks, cudaStream_t st) {
  if (a.N <= 0) return cudaSuccess;
  if (fp64) {
    // 8 lanes a row spend the fewest instructions; 16 hold half the rows a warp, so
    // twice the warps stay resident where the rows' columns fill the shared memory, and
    // more run where there are few rows (up to 32 an SM). us with 16 | 8 lanes: 30,000
    // rows x 121 trials, 40 ifg 208 | 153, 60 ifg 244 | 232, 100 ifg 349 | 362, 200 ifg
    // 731 | 1118, 256 ifg and 9 trials 635 | 1068; 3,000 rows x 20 ifg x 41 20.5 | 24.1
    const bool wide = a.M > 64 || a.N <= 2 * static_cast<int64_t>(grid_blocks);
    return wide ? launch_topofit_f64<16>(a, grid_blocks, st) : launch_topofit_f64<8>(a, grid_blocks, st);
  }
  return launch_topofit_f32(a, grid_blocks, st);
}

// ============================================================= finalize ===
// rms_difference + stop rule (:307-313, :2045-2057); when continuing, the
// P-square update (:364-381, :1642-1683) producing the prand_hi table that the
// next k_bin turns into weights. Sums use explicit _rn arithmetic and the
// reference's order so the table matches the reference given equal inputs.
//
// One block, bound by the latency of its serial parts: the operands are fetched
// together up front, the two ordered sums run in two warps at once, and an
// interpolated value adds only the 8 taps that meet a sample (the other 71
// multiply a zero). 33 -> 4.4 us a launch.
__device__ __forceinline__ void finalize_body(const FinalizeArgs& a) {
  __shared__ double sh[256];
  __shared__ double na[kCohBins], nr[kCohBins], prand[kCohBins], interp_in[kCohBins + 1], taps[80];
  __shared__ double num_s, den_s;
  __shared__ int go_on;
  const int tid = threadIdx.x;
  double st0 = 0.0, st1 = 0.0;
  int inv = 0;
  if (tid == 0) {
    st0 = a.state[0];
    st1 = a.state[1];
    inv = *a.n_invalid;
  }
  if (tid < kCohBins) {
    na[tid] = static_cast<double>(a.hist[tid]);
    nr[tid] = a.nr_scaled[tid];
  }
  if (tid >= 128 && tid < 128 + 79) taps[tid - 128] = a.taps79[tid - 128];
  double s = 0.0;
  for (int i0 = tid; i0 < a.n_partial; i0 += 256 * 10) {
    double v[10];
#pragma unroll
    for (int u = 0; u < 10; ++u) v[u] = i0 + 256 * u < a.n_partial ? a.rms_partial[i0 + 256 * u] : 0.0;
#pragma unroll
    for (int u = 0; u < 10; ++u)
      if (i0 + 256 * u < a.n_partial) s += v[u];
  }
  sh[tid] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (tid < w) sh[tid] += sh[tid + w];
    __syncthreads();
  }
  if (tid == 0) {
    const double rms = sqrt(sh[0] / static_cast<double>(a.N > 0 ? a.N : 1));
    const double gcs = st0;
    const double delta = rms - gcs;
    const int64_t i_loop = static_cast<int64_t>(st1);
    const int64_t cap = a.gamma_max_iterations > 1 ? a.gamma_max_iterations : 1;
    const bool stop = fabs(delta) < a.gamma_change_convergence || i_loop >= cap;
    a.state[0] = rms;
    a.state[1] = static_cast<double>(i_loop + 1);
    a.state[2] = rms;
    a.state[3] = delta;
    a.stats_out[0] = static_cast<double>(i_loop);
    a.stats_out[1] = rms;
    a.stats_out[2] = delta;
    a.stats_out[3] = stop ? 1.0 : 0.0;
    a.stats_out[4] = static_cast<double>(inv);
    go_on = ((!stop || a.force_continue) && a.psquare) ? 1 : 0;
    interp_in[0] = 1.0;
  } else if (tid == 32) {
    // Nr rescaled so its low-coherence mass matches Na's (sequential sums)
    double den = 0.0;
    for (int i = 0; i < a.low_coh_thresh; ++i) den = __dadd_rn(den, nr[i]);
    den_s = den;
  } else if (tid == 64) {
    double num = 0.0;
    for (int i = 0; i < a.low_coh_thresh; ++i) num = __dadd_rn(num, na[i]);
    num_s = num;
  }
  __syncthreads();
  if (!go_on) return;
  if (tid < kCohBins) {
    const double nrv = __dmul_rn(nr[tid], den_s > 0.0 ? num_s / den_s : 1.0);
    a.nr_scaled[tid] = nrv;
    const double d = na[tid] == 0.0 ? 1.0 : na[tid];
    double p = fmin(nrv / d, 1.0);
    if (tid < a.low_coh_thresh) p = 1.0;
    if (tid >= static_cast<int>(a.nr_max_nz_ix)) p = 0.0;
    prand[tid] = p;
  }
  __syncthreads();
  // lfilter(gausswin, [1]*7 ++ prand), shifted by 7, / sum(gausswin)
  if (tid < kCohBins) {
    const int ix = tid + 7;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      const int j = ix - k;
      const double v = j < 7 ? 1.0 : prand[j - 7];
      acc = __dadd_rn(acc, __dmul_rn(a.g7w[k], v));
    }
    interp_in[1 + tid] = acc / a.g7sum;
  }
  __syncthreads();
  // matlab_interp(.., 10) with the 79-tap FIR, delay 39, tail trimmed to 1001:
  // tap k meets sample (n - k) / 10 where that is whole, in tap order
  for (int i = tid; i < 1001; i += 256) {
    const int n = i + 39;
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = n % 10 + 10 * j, q = n / 10 - j;
      if (k < 79 && q >= 0 && q < 101) acc = __dadd_rn(acc, __dmul_rn(taps[k], interp_in[q]));
    }
    a.lut[i] = __dmul_rn(acc, 10.0);
  }
}

// In the graph that runs the loop to convergence this is the body's last node:
// it keeps the loop going while it has not raised the stop flag.
__global__ void __launch_bounds__(256) k_finalize(FinalizeArgs a) {
  finalize_body(a);
  if (a.set_loop && threadIdx.x == 0) cudaGraphSetConditional(a.loop, a.stats_out[3] == 0.0 ? 1u : 0u);
}

cudaError_t launch_finalize(const FinalizeArgs& a, cudaStream_t st) {
  k_finalize<<<1, 256, 0, st>>>(a);
  return cudaGetLastError();
}

// ========================================================= SNR weighting ==
// snr_weighting (:1875-1897) from the residual phase written by the last
// topofit: w = g / sqrt(0.5 (mean amp^2 - g^2)), g = mean(amp cos(ph_res)).
template <typename R>
__global__ void __launch_bounds__(256) k_snr_weight(const R* ph_res, const float* amp, int64_t N, int M, R* w_out) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t s = gw; s < N; s += nw) {
    double g = 0.0, a2 = 0.0;
    for (int c = lane; c < M; c += 32) {
      const double am = static_cast<double>(amp[s * M + c]);
      g += am * cos(static_cast<double>(ph_res[s * M + c]));
      a2 += am * am;
    }
    g = warp_sum(g);
    a2 = warp_sum(a2);
    if (lane == 0) {
      const double mm = static_cast<double>(M > 0 ? M : 1);
      g /= mm;
      a2 /= mm;
      const double sig = sqrt(0.5 * (a2 - g * g));
      w_out[s] = static_cast<R>(sig != 0.0 ? g / sig : 0.0);
    }
  }
}

cudaError_t launch_snr_weight(const TopoArgs& t, const float* amp, void* w_out, bool fp64, int sm_count,
                              cudaStream_t st) {
  const int blocks = sm_count * 8;
  if (fp64)
    k_snr_weight<double><<<blocks, 256, 0, st>>>(static_cast<const double*>(t.ph_res), amp, t.N, t.M,
                                                 static_cast<double*>(w_out));
  else
    k_snr_weight<float><<<blocks, 256, 0, st>>>(static_cast<const float*>(t.ph_res), amp, t.N, t.M,
                                                static_cast<float*>(w_out));
  return cudaGetLastError();
}

// ============================================== random-phase histogram ====
// random_coherence_histogram / topofit_phase_row_coh (:1310-1512) in FP64; every
// sum runs over the columns in the reference's order.
// The trial phasors e^{-j theta_c m} of every (column, trial), theta_c =
// (bp_c / range) * pi/4 (topofit_phase_row_coh, native_stage2.rs:1438-1470):
// the same for every random row, so they are evaluated once, [m][T].
__global__ void __launch_bounds__(256) k_trial_phasors(const double* __restrict__ bp, int m, int n_half,
                                                       double2* __restrict__ E) {
  const int T = 2 * n_half + 1;
  double mn = INFINITY, mx = -INFINITY;
  for (int c = 0; c < m; ++c) {
    mn = fmin(mn, bp[c]);
    mx = fmax(mx, bp[c]);
  }
  double range = mx - mn;
  if (range == 0.0) range = 1.0;
  const double qpi = 3.14159265358979323846 / 4.0;
  const int64_t total = static_cast<int64_t>(m) * T;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(idx / T), t = static_cast<int>(idx - static_cast<int64_t>(c) * T);
    double sn, cs;
    sincos(__dmul_rn(__dmul_rn(bp[c] / range, qpi), static_cast<double>(t - n_half)), &sn, &cs);
    E[idx] = make_double2(cs, sn);
  }
}

// A warp takes R rows: their trial sums run together (lanes over trials, each
// phasor of the table read once for R rows, columns in order), the trials ranked by
// |S|^2; a row whose two largest lie within rounding is decided by |S| / m as the
// reference compares it. The refinement's elementwise steps run over all elements
// of the R rows, its ordered sums side by side, one lane a chain (by themselves
// three chains of m dependent additions a row, the whole warp waiting). Bound by
// latency: two warps a scheduler (222 registers at R = 8) keep the FP64 pipe 43 %
// busy with 6 operations per (row, trial, column), issue 41 %. 300,000 rows x 60 x
// 161 trials: 4.4 -> 2.55 ms.
constexpr int kHistWarps = 4;
template <int R>
__global__ void __launch_bounds__(32 * kHistWarps) k_random_hist(
    const double* __restrict__ rnd, int64_t n_rand, const double* __restrict__ bp, int m,
    const int64_t* __restrict__ ia, const int64_t* __restrict__ ib, int small_baseline, int n_half, double cutoff0,
    double dbin, const double2* __restrict__ E, int32_t* hist) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  double2* u = reinterpret_cast<double2*>(smem_raw) + static_cast<int64_t>(wib) * R * m;
  double* ph = reinterpret_cast<double*>(reinterpret_cast<double2*>(smem_raw) + static_cast<int64_t>(kHistWarps) * R * m) +
               static_cast<int64_t>(wib) * R * m;
  __shared__ int sh_hist[kCohBins];
  __shared__ double sh_k[kHistWarps][R], sh_sum[kHistWarps][R][2];
  for (int i = tid; i < kCohBins; i += blockDim.x) sh_hist[i] = 0;
  __syncthreads();
  const int T = 2 * n_half + 1;
  double mn = INFINITY, mx = -INFINITY;
  for (int c = 0; c < m; ++c) {
    mn = fmin(mn, bp[c]);
    mx = fmax(mx, bp[c]);
  }
  double range = mx - mn;
  if (range == 0.0) range = 1.0;
  const double qpi = 3.14159265358979323846 / 4.0;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + tid) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  // the sum of one component of row r over the columns, in order, by lane 2 r + s
  auto ordered_sums = [&]() {
    __syncwarp();
    if (lane < 2 * R) {
      const double2* x = u + (lane >> 1) * m;
      double acc = 0.0;
      if (lane & 1)
        for (int c = 0; c < m; ++c) acc = __dadd_rn(acc, x[c].y);
      else
        for (int c = 0; c < m; ++c) acc = __dadd_rn(acc, x[c].x);
      sh_sum[wib][lane >> 1][lane & 1] = acc;
    }
    __syncwarp();
  };
  for (int64_t row0 = gw * R; row0 < n_rand; row0 += nw * R) {
    __syncwarp();
    // e^{j ph_c} of the rows (rows past the end repeat the last one)
    for (int idx = lane; idx < R * m; idx += 32) {
      const int c = idx / R, r = idx % R;
      const int64_t row = row0 + r < n_rand ? row0 + r : n_rand - 1;
      const double p = small_baseline ? rnd[row + ib[c] * n_rand] - rnd[row + ia[c] * n_rand] : rnd[row + c * n_rand];
      double sn, cs;
      sincos(p, &sn, &cs);
      ph[r * m + c] = p;
      u[r * m + c] = make_double2(cs, sn);
    }
    __syncwarp();
    Top2 top[R];
#pragma unroll
    for (int r = 0; r < R; ++r) top[r] = Top2{-1.0, -1.0, 0};
    for (int t0 = 0; t0 < T; t0 += 32) {
      const int rem = T - t0;
      if (rem * R <= 32) {
        // the last few trials: a lane for each (row, trial)
        constexpr int PER = 32 / R;
        const int rr = lane / PER, j = lane % PER, t = t0 + (j < rem ? j : 0);
        double sre = 0.0, sim = 0.0;
        for (int c = 0; c < m; ++c) {
          const double2 e = E[static_cast<int64_t>(c) * T + t], w = u[rr * m + c];
          sre = __dadd_rn(sre, __fma_rn(w.x, e.x, __dmul_rn(w.y, e.y)));
          sim = __dadd_rn(sim, __fma_rn(w.y, e.x, -__dmul_rn(w.x, e.y)));
        }
        const double sq = __fma_rn(sre, sre, __dmul_rn(sim, sim));
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (r == rr && j < rem) top[r].add(sq, t);
      } else {
        const int t = t0 + lane < T ? t0 + lane : T - 1;
        double sre[R], sim[R];
#pragma unroll
        for (int r = 0; r < R; ++r) sre[r] = sim[r] = 0.0;
#pragma unroll 4
        for (int c = 0; c < m; ++c) {
          const double2 e = E[static_cast<int64_t>(c) * T + t];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double2 w = u[r * m + c];
            sre[r] = __dadd_rn(sre[r], __fma_rn(w.x, e.x, __dmul_rn(w.y, e.y)));
            sim[r] = __dadd_rn(sim[r], __fma_rn(w.y, e.x, -__dmul_rn(w.x, e.y)));
          }
        }
        if (t0 + lane < T) {
#pragma unroll
          for (int r = 0; r < R; ++r) top[r].add(__fma_rn(sre[r], sre[r], __dmul_rn(sim[r], sim[r])), t);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(kFull, top[r].best, o), os = __shfl_xor_sync(kFull, top[r].second, o);
        const int ot = __shfl_xor_sync(kFull, top[r].t, o);
        const bool theirs = ob > top[r].best || (ob == top[r].best && ot < top[r].t);
        top[r].second = fmax(theirs ? top[r].best : ob, theirs ? os : top[r].second);
        if (theirs) {
          top[r].best = ob;
          top[r].t = ot;
        }
      }
      int bt = top[r].t;
      if (!(top[r].best - top[r].second > 1.0e-13 * top[r].best)) {
        // |S| / m as compared by the reference (topofit_phase_row_coh)
        double best = -1.0;
        bt = 0;
        for (int t = lane; t < T; t += 32) {
          double sre = 0.0, sim = 0.0;
          for (int c = 0; c < m; ++c) {
            const double2 e = E[static_cast<int64_t>(c) * T + t], w = u[r * m + c];
            sre = __dadd_rn(sre, __fma_rn(w.x, e.x, __dmul_rn(w.y, e.y)));
            sim = __dadd_rn(sim, __fma_rn(w.y, e.x, -__dmul_rn(w.x, e.y)));
          }
          const double v = hypot(sre, sim) / static_cast<double>(m);
          if (v > best) {
            best = v;
            bt = t;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(kFull, best, o);
          const int ot = __shfl_xor_sync(kFull, bt, o);
          if (ob > best || (ob == best && ot < bt)) {
            best = ob;
            bt = ot;
          }
        }
      }
      if (lane == 0) sh_k[wib][r] = qpi / range * static_cast<double>(bt - n_half);
    }
    __syncwarp();
    for (int idx = lane; idx < R * m; idx += 32) {
      const int r = idx / m, c = idx - r * m;
      double sn, cs;
      sincos(__dsub_rn(ph[idx], __dmul_rn(sh_k[wib][r], bp[c])), &sn, &cs);
      u[idx] = make_double2(cs, sn);
    }
    ordered_sums();
    for (int idx = lane; idx < R * m; idx += 32) {
      const int r = idx / m, c = idx - r * m;
      const double cs = u[idx].x, sn = u[idx].y, ore = sh_sum[wib][r][0], oim = sh_sum[wib][r][1];
      const double pre = __dsub_rn(__dmul_rn(cs, ore), __dmul_rn(sn, -oim));
      const double pim = __dadd_rn(__dmul_rn(cs, -oim), __dmul_rn(sn, ore));
      u[idx] = make_double2(__dmul_rn(bp[c], atan2(pim, pre)), __dmul_rn(bp[c], bp[c]));
    }
    ordered_sums();
    if (lane < R) {
      const double mopt = sh_sum[wib][lane][0];
      double den = sh_sum[wib][lane][1];
      if (den == 0.0) den = 1.0;
      sh_k[wib][lane] = sh_k[wib][lane] + mopt / den;
    }
    __syncwarp();
    for (int idx = lane; idx < R * m; idx += 32) {
      const int r = idx / m, c = idx - r * m;
      double sn, cs;
      sincos(__dsub_rn(ph[idx], __dmul_rn(sh_k[wib][r], bp[c])), &sn, &cs);
      u[idx] = make_double2(cs, sn);
    }
    ordered_sums();
    if (lane < R && row0 + lane < n_rand) {
      const double coh = hypot(sh_sum[wib][lane][0], sh_sum[wib][lane][1]) / static_cast<double>(m > 1 ? m : 1);
      const int b = coh_bin(coh, cutoff0, dbin);
      if (b >= 0) atomicAdd(&sh_hist[b], 1);
    }
  }
  __syncthreads();
  for (int i = tid; i < kCohBins; i += blockDim.x)
    if (sh_hist[i]) atomicAdd(&hist[i], sh_hist[i]);
}

template <int R>
static cudaError_t random_hist_rows(const double* rnd, int64_t n_rand, const double* bp, int m, const int64_t* ia,
                                    const int64_t* ib, int small_baseline, int n_half, double cutoff0, double dbin,
                                    const double2* phasors, int32_t* hist, int sm_count, cudaStream_t st) {
  const size_t sm = static_cast<size_t>(kHistWarps) * R * m * (sizeof(double2) + sizeof(double));
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  const int64_t per_block = static_cast<int64_t>(kHistWarps) * R;
  const int64_t blocks =
      std::max<int64_t>(1, std::min<int64_t>((n_rand + per_block - 1) / per_block, static_cast<int64_t>(sm_count) * 8));
  k_random_hist<R><<<static_cast<unsigned>(blocks), 32 * kHistWarps, sm, st>>>(
      rnd, n_rand, bp, m, ia, ib, small_baseline, n_half, cutoff0, dbin, phasors, hist);
  return cudaGetLastError();
}

cudaError_t launch_random_hist(const double* rnd, int64_t n_rand, const double* bp, int m, const int64_t* ia,
                               const int64_t* ib, int small_baseline, int n_half, double cutoff0, double dbin,
                               double2* phasors, int32_t* hist, int sm_count, cudaStream_t st) {
  const int64_t n_ph = static_cast<int64_t>(m) * (2 * n_half + 1);
  k_trial_phasors<<<static_cast<unsigned>(std::min<int64_t>((n_ph + 255) / 256, static_cast<int64_t>(sm_count) * 8)),
                    256, 0, st>>>(bp, m, n_half, phasors);
  // 8 rows a warp up to 64 columns (46 KB at 60; registers allow two blocks an SM), 4 beyond
  return m <= 64 ? random_hist_rows<8>(rnd, n_rand, bp, m, ia, ib, small_baseline, n_half, cutoff0, dbin, phasors, hist,
                                       sm_count, st)
                 : random_hist_rows<4>(rnd, n_rand, bp, m, ia, ib, small_baseline, n_half, cutoff0, dbin, phasors, hist,
                                       sm_count, st);
}


// ============================================================== stage 3 ===
// Stage-3 re-estimate (pystamps/pipeline/ported.py:4489-4550): for every grid
// cell holding a selected PS, the 32x32 patch of the stage-2 grid around it with
// the PS's own cell zeroed is CLAP-filtered (_clap_filt_patch, :992-1009) and
// the filtered value at that cell is kept; then each selected PS is re-fitted
// (_ps_topofit_single, :2355-2431) against it.

// np.exp(-1j * x) in complex64: (cos x, -sin x)
__device__ __forceinline__ float2 s3_cis_neg(float x) {
  float s, c;
  sincosf(x, &s, &c);
  return make_float2(c, -s);
}

struct S3Fit {
  float K, C, coh;
};

// _ps_topofit_refine_candidate (ported.py:2473-2508), float32, lanes over columns
__device__ S3Fit s3_refine(const float2* cpx, const float* bp, int n, double den_lin, double coarse_k0, int lane) {
  float K0 = static_cast<float>(coarse_k0);
  float ox = 0.f, oy = 0.f;
  for (int k = lane; k < n; k += 32) {
    const float2 r = cmul_rn(cpx[k], s3_cis_neg(__fmul_rn(K0, bp[k])));
    ox += r.x;
    oy += r.y;
  }
  ox = warp_sum(ox);
  oy = warp_sum(oy);
  float mo = 0.f;
  for (int k = lane; k < n; k += 32) {
    const float2 r = cmul_rn(cpx[k], s3_cis_neg(__fmul_rn(K0, bp[k])));
    const float2 q = cmul_rn(r, make_float2(ox, -oy));
    const float wgt = hypotf(cpx[k].x, cpx[k].y);
    mo += __fmul_rn(__fmul_rn(wgt, bp[k]), __fmul_rn(wgt, atan2f(q.y, q.x)));
  }
  mo = warp_sum(mo);
  K0 = __fadd_rn(K0, __fdiv_rn(mo, static_cast<float>(den_lin)));
  float mx = 0.f, my = 0.f, den = 0.f;
  for (int k = lane; k < n; k += 32) {
    const float2 r = cmul_rn(cpx[k], s3_cis_neg(__fmul_rn(K0, bp[k])));
    mx += r.x;
    my += r.y;
    den += hypotf(r.x, r.y);
  }
  mx = warp_sum(mx);
  my = warp_sum(my);
  den = warp_sum(den);
  if (den == 0.f) den = 1.f;
  return {K0, atan2f(my, mx), hypotf(mx, my) / den};
}

// One warp per selected PS: psdph against the re-estimated patch phase, the
// reference's invalid-row rule, then _ps_topofit_single with the near-max
// candidate rule (tolerance 2e-4), refinement of every candidate and the
// reference's choice among them.
__global__ void __launch_bounds__(128) k_s3_fit(S3FitArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int T = 2 * a.n_half + 1;
  const int nf = a.n_fit, M = a.M;
  unsigned char* base = smem_raw + static_cast<size_t>(wib) * a.warp_smem;
  float2* cpx = reinterpret_cast<float2*>(base);
  float* bp = reinterpret_cast<float*>(cpx + nf);
  float* tp = bp + nf;
  float* ct = tp + nf;
  const int64_t gw = static_cast<int64_t>(blockIdx.x) * 4 + wib;
  const int64_t nw = static_cast<int64_t>(gridDim.x) * 4;
  for (int64_t r = gw; r < a.n_sel; r += nw) {
    const int job = a.job_of[r];
    const int64_t row = a.row ? static_cast<int64_t>(a.row[r]) : r;  // row of ph / bp
    bool zero = false;
    for (int c = lane; c < M; c += 32) {
      const float2 pp = a.job_out[static_cast<int64_t>(job) * M + c];
      a.ph_patch2[r * M + c] = pp;
      a.ph_res2[r * M + c] = 0.f;
      const float2 h = a.ph[row * M + c];
      // psdph = ph * conj(ph_patch2) in f64 (exact products of f32 values)
      const double re = static_cast<double>(h.x) * pp.x + static_cast<double>(h.y) * pp.y;
      const double im = static_cast<double>(h.y) * pp.x - static_cast<double>(h.x) * pp.y;
      if (re == 0.0 && im == 0.0) zero = true;
    }
    if (__any_sync(0xffffffffu, zero)) {
      if (lane == 0) {
        a.K2[r] = __longlong_as_double(0x7ff8000000000000LL);
        a.coh2[r] = __longlong_as_double(0x7ff8000000000000LL);
        a.C2[r] = 0.0;
      }
      continue;
    }
    float mn = __int_as_float(0x7f800000), mx = -mn;
    for (int k = lane; k < nf; k += 32) {
      const int c = a.fit[k];
      const float2 pp = a.job_out[static_cast<int64_t>(job) * M + c];
      const float2 h = a.ph[row * M + c];
      const double re = static_cast<double>(h.x) * pp.x + static_cast<double>(h.y) * pp.y;
      const double im = static_cast<double>(h.y) * pp.x - static_cast<double>(h.x) * pp.y;
      const double mg = hypot(re, im);
      cpx[k] = make_float2(static_cast<float>(re / mg), static_cast<float>(im / mg));
      bp[k] = a.bp_row_inv ? a.bp[c] : a.bp[row * M + c];
      mn = fminf(mn, bp[k]);
      mx = fmaxf(mx, bp[k]);
    }
    mn = -warp_max(-mn);
    mx = warp_max(mx);
    double range = static_cast<double>(__fsub_rn(mx, mn));
    if (range == 0.0) range = 1.0;
    const float rf = static_cast<float>(range), qp = 0.785398163397448309615f;
    float den = 0.f, dl = 0.f;
    for (int k = lane; k < nf; k += 32) {
      tp[k] = __fmul_rn(__fdiv_rn(bp[k], rf), qp);
      const float ab = hypotf(cpx[k].x, cpx[k].y);
      const float wb = __fmul_rn(ab, bp[k]);
      den += ab;
      dl += __fmul_rn(wb, wb);
    }
    double denom = static_cast<double>(warp_sum(den));
    double den_lin = static_cast<double>(warp_sum(dl));
    if (denom == 0.0) denom = 1.0;
    if (den_lin == 0.0) den_lin = 1.0;
    __syncwarp();
    // coherence of every trial, columns summed in order (the reference adds
    // the rows of its (columns, trials) product one after another)
    float cmax = -1.f;
    for (int t = lane; t < T; t += 32) {
      const float tm = static_cast<float>(t - a.n_half);
      float sx = 0.f, sy = 0.f;
      for (int k = 0; k < nf; ++k) {
        const float2 p = cmul_rn(s3_cis_neg(__fmul_rn(tp[k], tm)), cpx[k]);
        sx = __fadd_rn(sx, p.x);
        sy = __fadd_rn(sy, p.y);
      }
      ct[t] = __fdiv_rn(hypotf(sx, sy), static_cast<float>(denom));
      cmax = fmaxf(cmax, ct[t]);
    }
    cmax = warp_max(cmax);
    __syncwarp();
    // candidates in trial order: local maxima within 2e-4 of the maximum
    int n_cand = 0, first = -1, last = -1, coarse_best = -1, refined_best = -1;
    S3Fit best_fit{0.f, 0.f, -1.f};
    float coarse_best_v = -1.f;
    for (int t0 = 0; t0 < T; t0 += 32) {
      const int t = t0 + lane;
      bool cand = false;
      if (t < T) {
        const float v = ct[t];
        bool lm;
        if (T == 1) lm = true;
        else if (t == 0) lm = v >= ct[1];
        else if (t == T - 1) lm = v >= ct[T - 2];
        else lm = v >= ct[t - 1] && v >= ct[t + 1];
        cand = lm && static_cast<double>(v) >= static_cast<double>(cmax) - 2.0e-4;
      }
      unsigned bal = __ballot_sync(0xffffffffu, cand);
      while (bal) {
        const int tt = t0 + __ffs(bal) - 1;
        bal &= bal - 1;
        if (first < 0) first = tt;
        last = tt;
        ++n_cand;
        if (ct[tt] > coarse_best_v) {
          coarse_best_v = ct[tt];
          coarse_best = tt;
        }
        const S3Fit f = s3_refine(cpx, bp, nf, den_lin, (3.14159265358979323846 / 4.0) / range * (tt - a.n_half), lane);
        if (static_cast<double>(f.coh) > static_cast<double>(best_fit.coh)) {
          best_fit = f;
          refined_best = tt;
        }
      }
    }
    int pick = refined_best;
    if (n_cand == 2 && first == 0 && last == T - 1) pick = coarse_best;
    if (pick < 0) pick = coarse_best >= 0 ? coarse_best : 0;  // refined coherences all NaN
    S3Fit f = best_fit;
    if (pick != refined_best)
      f = s3_refine(cpx, bp, nf, den_lin, (3.14159265358979323846 / 4.0) / range * (pick - a.n_half), lane);
    for (int k = lane; k < nf; k += 32) {
      const float2 res = cmul_rn(cpx[k], s3_cis_neg(__fmul_rn(f.K, bp[k])));
      a.ph_res2[r * M + a.fit[k]] = atan2f(res.y, res.x);
    }
    if (lane == 0) {
      a.K2[r] = static_cast<double>(f.K);
      a.C2[r] = static_cast<double>(f.C);
      a.coh2[r] = static_cast<double>(f.coh);
    }
    __syncwarp();
  }
}

cudaError_t launch_s3_fit(const S3FitArgs& a, int sm_count, cudaStream_t st) {
  if (a.n_sel <= 0) return cudaSuccess;
  const size_t sm = 4 * a.warp_smem;
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_s3_fit, 128, sm);
  if (e != cudaSuccess) return e;
  const int64_t blocks =
      std::min<int64_t>((a.n_sel + 3) / 4, static_cast<int64_t>(sm_count) * std::max(per_sm, 1));
  k_s3_fit<<<static_cast<unsigned>(blocks), 128, sm, st>>>(a);
  return cudaGetLastError();
}

// ================================================= registry topofit =======
// The registry's topofit (pystamps/kernels/accelerated.py:316-380 ->
// ported._ps_topofit_single, pystamps/pipeline/ported.py:2355-2431; the PyO3
// twin src/lib.rs:525-586 uses the same rule with tolerance 5e-3): per row,
// the non-zero columns only (zero columns take no part; an all-zero row gives
// NaN), trial coherences with columns summed in order, the near-max candidate
// set (local maxima within `tol` of the maximum), every candidate refined
// (_ps_topofit_refine_candidate, :2480-2513) and the reference's choice among
// them (_ps_topofit_select_candidate, :2451-2477). R is the row's real type:
// float for complex64 rows (the reference's single-precision path), double for
// complex128 rows. One warp per row.
template <typename R>
struct NearFit {
  R K, C, coh;
};

template <typename R>
__device__ __forceinline__ typename CT<R>::C cis_neg_r(R x) {
  R s, c;
  sincos_r(x, &s, &c);
  return mk(c, -s);
}

template <typename R>
__device__ NearFit<R> near_refine(const typename CT<R>::C* cv, const R* bv, int nf, R den_lin, double coarse_k0,
                                  int lane) {
  using C = typename CT<R>::C;
  R K0 = static_cast<R>(coarse_k0);
  R ox = 0, oy = 0;
  for (int k = lane; k < nf; k += 32) {
    const C r = cmul_rn(cv[k], cis_neg_r<R>(mul_rn(K0, bv[k])));
    ox = add_rn(ox, r.x);
    oy = add_rn(oy, r.y);
  }
  ox = warp_sum(ox);
  oy = warp_sum(oy);
  R mo = 0;
  for (int k = lane; k < nf; k += 32) {
    const C r = cmul_rn(cv[k], cis_neg_r<R>(mul_rn(K0, bv[k])));
    const C q = cmul_rn(r, mk(ox, -oy));
    const R wgt = hypot_r(cv[k].x, cv[k].y);
    mo = add_rn(mo, mul_rn(mul_rn(wgt, bv[k]), mul_rn(wgt, atan2_r(q.y, q.x))));
  }
  mo = warp_sum(mo);
  K0 = add_rn(K0, mo / den_lin);
  R mx = 0, my = 0, den = 0;
  for (int k = lane; k < nf; k += 32) {
    const C r = cmul_rn(cv[k], cis_neg_r<R>(mul_rn(K0, bv[k])));
    mx = add_rn(mx, r.x);
    my = add_rn(my, r.y);
    den = add_rn(den, hypot_r(r.x, r.y));
  }
  mx = warp_sum(mx);
  my = warp_sum(my);
  den = warp_sum(den);
  if (den == R(0)) den = R(1);
  return {K0, atan2_r(my, mx), hypot_r(mx, my) / den};
}

// Trial phasors of every (column, trial) for a baseline vector all rows share:
// a row without zero columns meets the same angles, so one sincos per table entry
// serves all of them (same expressions, same bits). 30,000 rows x 30 x 81 trials in
// FP64: 0.36 -> 0.15 ms.
template <typename R>
__global__ void __launch_bounds__(256) k_near_max_table(const R* __restrict__ bp, int M, int n_half,
                                                        typename CT<R>::C* __restrict__ E) {
  const int T = 2 * n_half + 1;
  R mn = bp[0], mx = bp[0];
  for (int k = 1; k < M; ++k) {
    mn = mn < bp[k] ? mn : bp[k];
    mx = mx > bp[k] ? mx : bp[k];
  }
  double range = static_cast<double>(add_rn(mx, -mn));
  if (range == 0.0) range = 1.0;
  const R range_r = static_cast<R>(range), qp = static_cast<R>(3.14159265358979323846 / 4.0);
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < M * T; idx += gridDim.x * blockDim.x) {
    const int c = idx / T, t = idx - c * T;
    E[idx] = cis_neg_r<R>(mul_rn(mul_rn(bp[c] / range_r, qp), static_cast<R>(t - n_half)));
  }
}

template <typename R>
__global__ void __launch_bounds__(32) k_topofit_near_max(NearMaxArgs a) {
  using C = typename CT<R>::C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x;
  const int M = a.M, T = 2 * a.n_half + 1;
  C* cv = reinterpret_cast<C*>(smem_raw);  // valid columns, compacted in column order
  R* bv = reinterpret_cast<R*>(cv + M);
  R* tp = bv + M;
  R* ct = tp + M;
  int* col = reinterpret_cast<int*>(ct + T);
  const C* cpx = static_cast<const C*>(a.cpx);
  const R* bp = static_cast<const R*>(a.bp);
  const C* __restrict__ E = static_cast<const C*>(a.table);
  const double nanv = __longlong_as_double(0x7ff8000000000000LL);
  for (int64_t r = blockIdx.x; r < a.n; r += gridDim.x) {
    int nf = 0;
    for (int c0 = 0; c0 < M; c0 += 32) {
      const int c = c0 + lane;
      C v = mk(R(0), R(0));
      R b = 0;
      bool valid = false;
      if (c < M) {
        v = cpx[r * M + c];
        b = a.bp_row_inv ? bp[c] : bp[r * M + c];
        valid = !(v.x == R(0) && v.y == R(0));  // complex != 0 (NaN parts count as non-zero)
        if (a.residual) a.residual[r * M + c] = make_float2(0.f, 0.f);
      }
      const unsigned bal = __ballot_sync(kFull, valid);
      if (valid) {
        const int k = nf + __popc(bal & ((1u << lane) - 1u));
        cv[k] = v;
        bv[k] = b;
        col[k] = c;
      }
      nf += __popc(bal);
    }
    __syncwarp();
    if (nf == 0) {
      if (lane == 0) a.K[r] = a.C[r] = a.coh[r] = nanv;
      continue;
    }
    R mn = bv[0], mx = bv[0];
    for (int k = lane; k < nf; k += 32) {
      mn = mn < bv[k] ? mn : bv[k];
      mx = mx > bv[k] ? mx : bv[k];
    }
    mn = warp_min(mn);
    mx = warp_max(mx);
    double range = static_cast<double>(add_rn(mx, -mn));
    if (range == 0.0) range = 1.0;
    const R range_r = static_cast<R>(range), qp = static_cast<R>(3.14159265358979323846 / 4.0);
    R den = 0, dl = 0;
    for (int k = lane; k < nf; k += 32) {
      tp[k] = mul_rn(bv[k] / range_r, qp);
      const R ab = hypot_r(cv[k].x, cv[k].y);
      const R wb = mul_rn(ab, bv[k]);
      den = add_rn(den, ab);
      dl = add_rn(dl, mul_rn(wb, wb));
    }
    R denom = warp_sum(den), den_lin = warp_sum(dl);
    if (denom == R(0)) denom = R(1);
    if (den_lin == R(0)) den_lin = R(1);
    __syncwarp();
    // coherence of every trial, columns summed in order
    R cmax = -1;
    for (int t = lane; t < T; t += 32) {
      const R tm = static_cast<R>(t - a.n_half);
      R sx = 0, sy = 0;
      if (E && nf == M) {
#pragma unroll 4
        for (int k = 0; k < nf; ++k) {
          const C p = cmul_rn(E[k * T + t], cv[k]);
          sx = add_rn(sx, p.x);
          sy = add_rn(sy, p.y);
        }
      } else {
        for (int k = 0; k < nf; ++k) {
          const C p = cmul_rn(cis_neg_r<R>(mul_rn(tp[k], tm)), cv[k]);
          sx = add_rn(sx, p.x);
          sy = add_rn(sy, p.y);
        }
      }
      ct[t] = hypot_r(sx, sy) / denom;
      cmax = cmax > ct[t] ? cmax : ct[t];
    }
    cmax = warp_max(cmax);
    __syncwarp();
    int n_cand = 0, first = -1, last = -1, coarse_best = -1, refined_best = -1;
    NearFit<R> best_fit{0, 0, -1};
    R coarse_best_v = -1;
    for (int t0 = 0; t0 < T; t0 += 32) {
      const int t = t0 + lane;
      bool cand = false;
      if (t < T) {
        const R v = ct[t];
        bool lm;
        if (T == 1) lm = true;
        else if (t == 0) lm = v >= ct[1];
        else if (t == T - 1) lm = v >= ct[T - 2];
        else lm = v >= ct[t - 1] && v >= ct[t + 1];
        cand = lm && static_cast<double>(v) >= static_cast<double>(cmax) - a.tol;
      }
      unsigned bal = __ballot_sync(kFull, cand);
      while (bal) {
        const int tt = t0 + __ffs(bal) - 1;
        bal &= bal - 1;
        if (first < 0) first = tt;
        last = tt;
        ++n_cand;
        if (ct[tt] > coarse_best_v) {
          coarse_best_v = ct[tt];
          coarse_best = tt;
        }
        const NearFit<R> f =
            near_refine<R>(cv, bv, nf, den_lin, (3.14159265358979323846 / 4.0) / range * (tt - a.n_half), lane);
        if (static_cast<double>(f.coh) > static_cast<double>(best_fit.coh)) {
          best_fit = f;
          refined_best = tt;
        }
      }
    }
    if (n_cand == 0) {  // no local maximum within tol (NaN coherences): np.argmax (a NaN wins)
      for (int t = 0; t < T; ++t) {
        if (isnan(ct[t])) {
          coarse_best = t;
          break;
        }
        if (ct[t] > coarse_best_v) {
          coarse_best_v = ct[t];
          coarse_best = t;
        }
      }
      if (coarse_best < 0) coarse_best = 0;
    }
    int pick = refined_best;
    if (n_cand <= 1 || (n_cand == 2 && first == 0 && last == T - 1)) pick = coarse_best;
    if (pick < 0) pick = coarse_best >= 0 ? coarse_best : 0;
    NearFit<R> f = best_fit;
    if (pick != refined_best)
      f = near_refine<R>(cv, bv, nf, den_lin, (3.14159265358979323846 / 4.0) / range * (pick - a.n_half), lane);
    if (a.residual)
      for (int k = lane; k < nf; k += 32) {
        const C res = cmul_rn(cv[k], cis_neg_r<R>(mul_rn(f.K, bv[k])));
        a.residual[r * M + col[k]] = make_float2(static_cast<float>(res.x), static_cast<float>(res.y));
      }
    if (lane == 0) {
      a.K[r] = static_cast<double>(f.K);
      a.C[r] = static_cast<double>(f.C);
      a.coh[r] = static_cast<double>(f.coh);
    }
    __syncwarp();
  }
}

size_t topofit_near_max_table(bool fp64, bool row_inv, int64_t n, int M, int n_half) {
  const int64_t entries = static_cast<int64_t>(M) * (2 * n_half + 1);
  // 64 rows pay for the table; 2^20 entries (16 MB of double2) still sit in L2
  if (!row_inv || n < 64 || entries > (int64_t(1) << 20)) return 0;
  return static_cast<size_t>(entries) * (fp64 ? sizeof(double2) : sizeof(float2));
}

size_t topofit_near_max_smem(bool fp64, int M, int n_half) {
  const size_t rs = fp64 ? sizeof(double) : sizeof(float);
  return static_cast<size_t>(M) * (2 * rs + rs + rs + sizeof(int)) + static_cast<size_t>(2 * n_half + 1) * rs + 16;
}

cudaError_t launch_topofit_near_max(const NearMaxArgs& a, bool fp64, int sm_count, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const size_t sm = topofit_near_max_smem(fp64, a.M, a.n_half);
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min<int64_t>(a.n, static_cast<int64_t>(sm_count) * 32);
  if (a.table) {
    const int n_e = a.M * (2 * a.n_half + 1);
    const unsigned tb = static_cast<unsigned>(std::min((n_e + 255) / 256, sm_count * 4));
    if (fp64)
      k_near_max_table<double><<<tb, 256, 0, st>>>(static_cast<const double*>(a.bp), a.M, a.n_half,
                                                   static_cast<double2*>(a.table));
    else
      k_near_max_table<float><<<tb, 256, 0, st>>>(static_cast<const float*>(a.bp), a.M, a.n_half,
                                                  static_cast<float2*>(a.table));
  }
  if (fp64)
    k_topofit_near_max<double><<<static_cast<unsigned>(blocks), 32, sm, st>>>(a);
  else
    k_topofit_near_max<float><<<static_cast<unsigned>(blocks), 32, sm, st>>>(a);
  return cudaGetLastError();
}

// ================================================ histogram with centers ==
// The registry's stage2_histogram (pystamps/kernels/accelerated.py:235-265):
// equally spaced centres use the ceil rule 1 + max(0, min(nc-1,
// ceil((v - cutoff0) / d))); otherwise the bin is searchsorted(mids, v,
// 'left') clipped to [0, nc-1]. Non-finite values are skipped. Integer
// atomics: the counts do not depend on the order.
__global__ void __launch_bounds__(256) k_hist_centers(const double* __restrict__ v, int64_t n,
                                                      const double* __restrict__ mids, int nc, int equal, double d,
                                                      double cutoff0, unsigned long long* __restrict__ counts) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double s = v[i];
    if (!isfinite(s)) continue;
    int b;
    if (equal) {
      const double q = ceil((s - cutoff0) / d);
      b = static_cast<int>(fmax(0.0, fmin(static_cast<double>(nc - 1), q)));
    } else {
      int lo = 0, hi = nc - 1;  // first of the nc-1 mids that is >= s
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (mids[mid] < s) lo = mid + 1;
        else hi = mid;
      }
      b = lo;
    }
    atomicAdd(&counts[b], 1ull);
  }
}

cudaError_t launch_hist_centers(const double* v, int64_t n, const double* mids, int nc, int equal, double d,
                                double cutoff0, unsigned long long* counts, int sm_count, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 255) / 256, static_cast<int64_t>(sm_count) * 8);
  k_hist_centers<<<static_cast<unsigned>(blocks), 256, 0, st>>>(v, n, mids, nc, equal, d, cutoff0, counts);
  return cudaGetLastError();
}

// ============================================================== batches ===
// Many patches, each iteration one launch per step over every active patch.
// Work units are numbered patch after patch (prefix tables); a unit finds its
// patch by binary search. Each unit runs the single-patch code on its patch's
// arguments, so a patch's results do not depend on what it is batched with.

// k_iter_begin over the active patches: their statistics cleared (a block per
// patch), K[1] <- K[0] and the P-square weights from iteration 2 on (elements
// numbered patch after patch over the whole grid). A block per patch copying its
// K took 0.22 ms an iteration of 12 patches of up to 200,000 PS, and the weights
// were looked up by every lane of every interferogram chunk of the binning.
__global__ void __launch_bounds__(256) k_batch_begin(BatchArgs b) {
  for (int p = blockIdx.x; p < b.P; p += gridDim.x) {
    if (!b.active[p]) continue;
    const PatchDev& d = b.patch[p];
    for (int i = threadIdx.x; i < kCohBins; i += blockDim.x) d.topo.hist[i] = 0;
    if (threadIdx.x == 0) *d.topo.n_invalid = 0;
    for (int i = threadIdx.x; i < d.fin.n_partial; i += blockDim.x) d.topo.rms_partial[i] = 0.0;
  }
  const int64_t total = b.ps_prefix[b.P];
  for (int64_t u = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < total;
       u += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int p = find_patch(b.ps_prefix, b.P, u);
    if (!b.active[p]) continue;
    const PatchDev& d = b.patch[p];
    const int64_t s = u - b.ps_prefix[p];
    d.K1[s] = static_cast<const float*>(d.bin.K)[s];
    if (d.psquare && d.fin.state[1] > 1.0)
      static_cast<float*>(d.bin.w)[s] = psquare_weight<float>(d.bin, static_cast<const float*>(d.bin.coh)[s]);
  }
}

__global__ void __launch_bounds__(256) k_batch_bin(BatchArgs b) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t total = b.bin_prefix[b.P];
  for (int64_t u = gw; u < total; u += nw) {
    const int p = find_patch(b.bin_prefix, b.P, u);
    if (!b.active[p]) continue;
    bin_task<float>(b.patch[p].bin, u - b.bin_prefix[p], lane);
  }
}

__global__ void __launch_bounds__(256) k_batch_overlap(BatchArgs b) {
  const int64_t total = b.ov_prefix[b.P];
  for (int64_t u = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < total;
       u += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int p = find_patch(b.ov_prefix, b.P, u);
    if (!b.active[p]) continue;
    overlap_any<float>(b.patch[p].ov, u - b.ov_prefix[p]);
  }
}

__global__ void __launch_bounds__(256) k_batch_finalize(BatchArgs b) {
  const int p = blockIdx.x;
  if (p >= b.P || !b.active[p]) return;
  const FinalizeArgs& f = b.patch[p].fin;
  finalize_body(f);
  __syncthreads();
  if (threadIdx.x == 0 && f.stats_out[3] != 0.0 && !f.force_continue) {
    b.active[p] = 0;
    atomicSub(b.n_active, 1);
  }
}

__global__ void k_batch_continue(cudaGraphConditionalHandle h, const int* n_active) {
  if (threadIdx.x == 0) cudaGraphSetConditional(h, *n_active > 0 ? 1u : 0u);
}

cudaError_t launch_batch_begin(const BatchArgs& b, int64_t total_ps, int sm_count, cudaStream_t st) {
  const int64_t blocks =
      std::max<int64_t>(1, std::min<int64_t>((total_ps + 255) / 256, static_cast<int64_t>(sm_count) * 8));
  k_batch_begin<<<static_cast<unsigned>(blocks), 256, 0, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_batch_bin(const BatchArgs& b, int64_t total, int sm_count, cudaStream_t st) {
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((total + 7) / 8, static_cast<int64_t>(sm_count) * 16));
  k_batch_bin<<<static_cast<unsigned>(blocks), 256, 0, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_batch_overlap(const BatchArgs& b, int64_t total, int sm_count, cudaStream_t st) {
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, static_cast<int64_t>(sm_count) * 32));
  k_batch_overlap<<<static_cast<unsigned>(blocks), 256, 0, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_batch_finalize(const BatchArgs& b, cudaStream_t st) {
  k_batch_finalize<<<b.P, 256, 0, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_batch_continue(cudaGraphConditionalHandle h, const int* n_active, cudaStream_t st) {
  k_batch_continue<<<1, 32, 0, st>>>(h, n_active);
  return cudaGetLastError();
}

// ============================================================== adjoints ==
// Differentiable stage-2 coherence with K given (no trial search):
//   grid  = bin(ph e^{-j K bp} w)              (k_bin, mode 0)
//   filt  = CLAP(grid; alpha, beta)            (k_clap + k_overlap)
//   p     = filt[cell] / |filt[cell]|          (resample + normalise)
//   gamma = |sum_c conj(p_c) ph_c e^{-j K bp_c}| / sum_c |conj(p_c) ph_c|
// Gradients use the complex convention g = dL/dRe + j dL/dIm. CLAP's window
// spectra are recomputed in the backward pass, not stored. R is the working
// precision (the context's): inputs arrive as float and are widened.

template <typename R>
__device__ __forceinline__ typename CT<R>::C unit_or_zero(const typename CT<R>::C f, R* mag) {
  const R m = hypot_r(f.x, f.y);
  *mag = m;
  return m != R(0) ? mk(f.x / m, f.y / m) : mk(R(0), R(0));
}

template <typename R>
__device__ __forceinline__ R row_bp(const CohArgs& a, int64_t s, int c) {
  return a.bp_row_inv ? static_cast<R>(a.bp[c]) : static_cast<R>(a.bp[s * a.M + c]);
}

template <typename R>
__device__ __forceinline__ typename CT<R>::C load_ph(const CohArgs& a, int64_t s, int c) {
  const float2 v = a.ph[s * a.M + c];
  return mk(static_cast<R>(v.x), static_cast<R>(v.y));
}

// S = sum_c conj(p_c) ph_c e^{-j K bp_c} and D = sum_c |conj(p_c) ph_c| of one PS (whole warp)
template <typename R>
__device__ __forceinline__ void coh_sums(const CohArgs& a, int64_t s, int lane, R* sx_o, R* sy_o, R* d_o) {
  using C = typename CT<R>::C;
  const C* __restrict__ filt = static_cast<const C*>(a.filt);
  const int64_t cell = a.cell_of[s];
  const R k = static_cast<const R*>(a.K)[s];
  R sx = R(0), sy = R(0), d = R(0);
  for (int c = lane; c < a.M; c += 32) {
    R mag;
    const C pp = unit_or_zero<R>(filt[cell * a.Mp + c], &mag);
    const C z = cmul(mk(pp.x, -pp.y), load_ph<R>(a, s, c));
    R sn, cs;
    sincos_r(k * row_bp<R>(a, s, c), &sn, &cs);
    const C r = cmul(z, mk(cs, -sn));
    sx += r.x;
    sy += r.y;
    d += hypot_r(z.x, z.y);
  }
  *sx_o = warp_sum(sx);
  *sy_o = warp_sum(sy);
  *d_o = warp_sum(d);
}

template <typename R>
__global__ void __launch_bounds__(256) k_coh_fwd(CohArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t s = gw; s < a.N; s += nw) {
    R sx, sy, d;
    coh_sums<R>(a, s, lane, &sx, &sy, &d);
    if (lane == 0) a.coh[s] = static_cast<float>(hypot_r(sx, sy) / (d != R(0) ? d : R(1)));
  }
}

template <typename R>
__global__ void __launch_bounds__(256) k_coh_bwd(CohArgs a) {
  using C = typename CT<R>::C;
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const C* __restrict__ filt = static_cast<const C*>(a.filt);
  C* __restrict__ gph = static_cast<C*>(a.gph);
  C* __restrict__ gf_out = static_cast<C*>(a.gf);
  for (int64_t s = gw; s < a.N; s += nw) {
    R sx, sy, d;
    coh_sums<R>(a, s, lane, &sx, &sy, &d);
    const int64_t cell = a.cell_of[s];
    const R k = static_cast<const R*>(a.K)[s];
    const R dd = d != R(0) ? d : R(1);
    const R sm = hypot_r(sx, sy);
    const R g = static_cast<R>(a.gcoh[s]);
    const R gam = sm / dd;
    // d gamma / d S = S / (|S| D); d gamma / d |z_c| = -gamma / D
    const C gS = sm > R(0) ? mk(g * sx / (sm * dd), g * sy / (sm * dd)) : mk(R(0), R(0));
    const R gD = -g * gam / dd;
    R gk = R(0);
    for (int c = lane; c < a.M; c += 32) {
      R mag;
      const C pp = unit_or_zero<R>(filt[cell * a.Mp + c], &mag);
      const C h = load_ph<R>(a, s, c);
      const C z = cmul(mk(pp.x, -pp.y), h);
      const R b = row_bp<R>(a, s, c);
      R sn, cs;
      sincos_r(k * b, &sn, &cs);
      const C e = mk(cs, -sn);
      const C r = cmul(z, e);
      // r = z e:  g_z = conj(e) g_S (+ the denominator term);  dr/dK = -j bp r
      C gz = cmul(mk(e.x, -e.y), gS);
      const R zm = hypot_r(z.x, z.y);
      if (zm > R(0)) {
        gz.x += gD * z.x / zm;
        gz.y += gD * z.y / zm;
      }
      gk += gS.x * (b * r.y) + gS.y * (-b * r.x);
      // z = conj(p) h:  g_h = p g_z,  g_p = conj(g_z) h
      gph[s * a.M + c] = cmul(pp, gz);
      const C gp = cmul(mk(gz.x, -gz.y), h);
      // p = f / |f|:  g_f = (g_p - p Re(conj(p) g_p)) / |f|
      C gf = mk(R(0), R(0));
      if (mag > R(0)) {
        const R rp = pp.x * gp.x + pp.y * gp.y;
        gf = mk((gp.x - pp.x * rp) / mag, (gp.y - pp.y * rp) / mag);
      }
      gf_out[s * a.M + c] = gf;
    }
    gk = warp_sum(gk);
    if (lane == 0) static_cast<R*>(a.gK)[s] = gk;
  }
}

// bin backward: grid[cell, c] += a ph with a = e^{-j K bp} w
template <typename R>
__global__ void __launch_bounds__(256) k_bin_bwd(CohArgs a) {
  using C = typename CT<R>::C;
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const C* __restrict__ ggrid = static_cast<const C*>(a.ggrid);
  C* __restrict__ gph = static_cast<C*>(a.gph);
  for (int64_t s = gw; s < a.N; s += nw) {
    const int64_t cell = a.cell_of[s];
    const R k = static_cast<const R*>(a.K)[s], w = static_cast<const R*>(a.w)[s];
    R gk = R(0);
    for (int c = lane; c < a.M; c += 32) {
      const R b = row_bp<R>(a, s, c);
      R sn, cs;
      sincos_r(-(b * k), &sn, &cs);
      const C co = mk(cs * w, sn * w);
      const C gg = ggrid[cell * a.Mp + c];
      const C gh = cmul(mk(co.x, -co.y), gg);
      const C prev = gph[s * a.M + c];
      gph[s * a.M + c] = mk(prev.x + gh.x, prev.y + gh.y);
      const C v = cmul(co, load_ph<R>(a, s, c));  // d(a h)/dK = -j bp a h
      gk += gg.x * (b * v.y) + gg.y * (-b * v.x);
    }
    gk = warp_sum(gk);
    if (lane == 0) static_cast<R*>(a.gK)[s] += gk;
  }
}

// per-cell sum of complex rows [N, M] in cell order (rows of one cell are
// contiguous), sequential in row order: d L / d filt from d L / d p_c
template <typename R>
__global__ void __launch_bounds__(256) k_cell_sum(CohArgs a, const int32_t* __restrict__ cell_start, int64_t G,
                                                  int nchunk, void* out_v) {
  using C = typename CT<R>::C;
  const C* __restrict__ src = static_cast<const C*>(a.gf);
  C* __restrict__ out = static_cast<C*>(out_v);
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t task = gw; task < G * nchunk; task += nw) {
    const int64_t cell = task / nchunk;
    const int c = static_cast<int>(task - cell * nchunk) * 32 + lane;
    R ax = R(0), ay = R(0);
    if (c < a.M) {
      for (int s = cell_start[cell]; s < cell_start[cell + 1]; ++s) {
        const C v = src[static_cast<int64_t>(s) * a.M + c];
        ax += v.x;
        ay += v.y;
      }
    }
    if (c < a.Mp) out[cell * a.Mp + c] = mk(ax, ay);
  }
}

template <typename R>
static cudaError_t coh_launch(const CohArgs& a, int which, int sm_count, cudaStream_t st) {
  int64_t blocks = (a.N + 7) / 8;
  if (blocks > static_cast<int64_t>(sm_count) * 16) blocks = static_cast<int64_t>(sm_count) * 16;
  if (blocks < 1) blocks = 1;
  if (which == 0)
    k_coh_fwd<R><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  else if (which == 1)
    k_coh_bwd<R><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  else
    k_bin_bwd<R><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_coh(const CohArgs& a, int which, bool fp64, int sm_count, cudaStream_t st) {
  return fp64 ? coh_launch<double>(a, which, sm_count, st) : coh_launch<float>(a, which, sm_count, st);
}

cudaError_t launch_cell_sum(const CohArgs& a, const int32_t* cell_start, int64_t G, void* out, bool fp64,
                            int sm_count, cudaStream_t st) {
  const int nchunk = (a.M + 31) / 32;
  int64_t blocks = (G * nchunk + 7) / 8;
  if (blocks > static_cast<int64_t>(sm_count) * 16) blocks = static_cast<int64_t>(sm_count) * 16;
  if (blocks < 1) blocks = 1;
  if (fp64)
    k_cell_sum<double><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a, cell_start, G, nchunk, out);
  else
    k_cell_sum<float><<<static_cast<unsigned>(blocks), 256, 0, st>>>(a, cell_start, G, nchunk, out);
  return cudaGetLastError();
}

template <typename R>
struct ClapBwdTile {
  R re[32][33];
  R im[32][33];
  R hs[32][33];
  R gre[32][33];
  R gim[32][33];
  R pad[8];
};

template <typename R>
__global__ void __launch_bounds__(128) k_clap_bwd(ClapBwdArgs b, typename CT<R>::Tw tw) {
  using C = typename CT<R>::C;
  const ClapArgs& a = b.f;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ClapBwdTile<R>* tiles = reinterpret_cast<ClapBwdTile<R>*>(smem_raw);
  R* lp = reinterpret_cast<R*>(tiles + 4);
  R* wt = lp + 1024;
  C* twf = reinterpret_cast<C*>(wt + 1024);
  C* twi = twf + 16;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nw = a.n_win, nw2 = nw * nw;
  for (int i = tid; i < 1024; i += 128) lp[i] = static_cast<R>(a.low_pass[i]);
  for (int i = tid; i < nw2; i += 128) wt[i] = static_cast<R>(a.wscaled[i]);
  if (tid < 16) {
    twf[tid] = tw.w[tid];
    twi[tid] = mk(tw.w[tid].x, -tw.w[tid].y);
  }
  R g7[7];
#pragma unroll
  for (int i = 0; i < 7; ++i) g7[i] = static_cast<R>(a.g7[i]);
  const int n_inc = nw / 4 > 1 ? nw / 4 : 1;
  const int ngroups = a.Mp / 4;
  const int64_t ntask = static_cast<int64_t>(a.nwi) * a.nwj * ngroups;
  const C* __restrict__ grid = static_cast<const C*>(a.grid);
  const C* __restrict__ gfilt = static_cast<const C*>(b.gfilt);
  C* __restrict__ wgrad = static_cast<C*>(b.wgrad);
  ClapBwdTile<R>& T = tiles[warp];
  const R alpha = static_cast<R>(a.alpha), beta = static_cast<R>(a.beta);
  double ga_acc = 0.0, gb_acc = 0.0;
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    const int64_t wi = task / ngroups;
    const int g = static_cast<int>(task - wi * ngroups);
    const int ix1 = static_cast<int>(wi / a.nwj), ix2 = static_cast<int>(wi - static_cast<int64_t>(ix1) * a.nwj);
    int i1 = ix1 * n_inc, rs = 0;
    if (i1 + nw > a.n_i) {
      rs = i1 + nw - a.n_i;
      i1 = a.n_i - nw;
    }
    int j1 = ix2 * n_inc, cs = 0;
    if (j1 + nw > a.n_j) {
      cs = j1 + nw - a.n_j;
      j1 = a.n_j - nw;
    }
    __syncthreads();
    for (int idx = tid; idx < 4 * 32 * 32; idx += 128) {
      const int q = idx >> 10, e = idx & 1023, r = e >> 5, cc = e & 31;
      if (r >= nw || cc >= nw) {
        tiles[q].re[r][cc] = R(0);
        tiles[q].im[r][cc] = R(0);
        tiles[q].gre[r][cc] = R(0);
        tiles[q].gim[r][cc] = R(0);
      }
    }
    for (int idx = tid; idx < nw2 * 4; idx += 128) {
      const int pix = idx >> 2, q = idx & 3;
      const int li = pix / nw, lj = pix - li * nw;
      const int c = 4 * g + q;
      C v = mk(R(0), R(0)), gy = mk(R(0), R(0));
      if (c < a.M) {
        const int64_t cell = static_cast<int64_t>(i1 + li) * a.n_j + (j1 + lj);
        v = grid[cell * a.Mp + c];
        if (isnan(v.x) || isnan(v.y)) v = mk(R(0), R(0));
        const R wv = (li < rs || lj < cs) ? R(0) : wt[(li - rs) * nw + (lj - cs)];
        const C go = gfilt[cell * a.Mp + c];
        gy = mk(go.x * wv, go.y * wv);  // out += w y  =>  g_y = w g_out
      }
      tiles[q].re[li][lj] = v.x;
      tiles[q].im[li][lj] = v.y;
      tiles[q].gre[li][lj] = gy.x;
      tiles[q].gim[li][lj] = gy.y;
    }
    __syncthreads();
    if (4 * g + warp < a.M) {
      // recompute the forward spectrum X = FFT2(x) and the smoothed magnitude
      if (lane < nw) fft_pass<R>(T.re, T.im, twf, lane, true);
      __syncwarp();
      fft_pass<R>(T.re, T.im, twf, lane, false);
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const R xr = T.re[k][lane], xi = T.im[k][lane];
        T.hs[k][lane] = sqrt(xr * xr + xi * xi);
      }
      __syncwarp();
      R t[32];
      const int sj = (lane + 16) & 31;
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        R acc = R(0);
#pragma unroll
        for (int d = -3; d <= 3; ++d)
          if (sj + d >= 0 && sj + d < 32) acc += T.hs[k][(lane + d) & 31] * g7[d + 3];
        t[k] = acc;
      }
      R o[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int sk = (k + 16) & 31;
        R acc = R(0);
#pragma unroll
        for (int d = -3; d <= 3; ++d)
          if (sk + d >= 0 && sk + d < 32) acc += t[(k + d) & 31] * g7[d + 3];
        o[k] = acc;
      }
      R v0, v1;
      const R med = warp_median1024_pair<R>(o, &T.hs[0][0], v0, v1);
      // g_Y = FFT2(g_y) (adjoint of the unnormalised inverse FFT)
      if (lane < nw) fft_pass<R>(T.gre, T.gim, twf, lane, true);
      __syncwarp();
      fft_pass<R>(T.gre, T.gim, twf, lane, false);
      const R inv_med = med != R(0) ? R(1) / med : R(1);
      R gmed = R(0), ga = R(0), gb = R(0);
      // t becomes dL/d(smoothed |X|), starting with the direct term
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const R xr = T.re[k][lane], xi = T.im[k][lane];
        const R gyr = T.gre[k][lane], gyi = T.gim[k][lane];
        const R hn = o[k] * inv_med;
        const R pw = a.alpha_is_one ? hn : pow(hn, alpha);
        const bool act = pw - R(1) > R(0);
        const R G = (act ? pw - R(1) : R(0)) * beta + lp[k * 32 + lane];
        const R gG = xr * gyr + xi * gyi;
        R ghn = R(0);
        if (act) {
          ghn = gG * beta * (a.alpha_is_one ? R(1) : alpha * pow(hn, alpha - R(1)));
          gb += gG * (pw - R(1));
          ga += gG * beta * pw * log(hn);
        }
        if (med != R(0)) gmed += ghn * (-o[k] * inv_med * inv_med);
        t[k] = med != R(0) ? ghn * inv_med : ghn;
        T.gre[k][lane] = gyr * G;  // g_X from Y = X G
        T.gim[k][lane] = gyi * G;
      }
      gmed = warp_sum(gmed);
      ga = warp_sum(ga);
      gb = warp_sum(gb);
      if (med != R(0)) {
        // med = (v0 + v1) / 2 of the smoothed magnitudes; ties share evenly
        int c0 = 0, c1 = 0;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          c0 += o[k] == v0 ? 1 : 0;
          c1 += o[k] == v1 ? 1 : 0;
        }
        c0 = warp_sum(c0);
        c1 = warp_sum(c1);
        const R share0 = v0 == v1 ? gmed / static_cast<R>(c0) : R(0.5) * gmed / static_cast<R>(c0);
        const R share1 = v0 == v1 ? R(0) : R(0.5) * gmed / static_cast<R>(c1);
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          if (o[k] == v0)
            t[k] += share0;
          else if (o[k] == v1)
            t[k] += share1;
        }
      }
      // adjoint of the separable smoothing: along k in registers, then across lanes
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int sk = (k + 16) & 31;
        R acc = R(0);
#pragma unroll
        for (int d = -3; d <= 3; ++d)
          if (sk + d >= 0 && sk + d < 32) acc += t[(k + d) & 31] * g7[d + 3];
        o[k] = acc;
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 32; ++k) T.hs[k][lane] = o[k];
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        R acc = R(0);
#pragma unroll
        for (int d = -3; d <= 3; ++d)
          if (sj + d >= 0 && sj + d < 32) acc += T.hs[k][(lane + d) & 31] * g7[d + 3];
        // H = |X|:  g_X += g_H X / |X|
        const R xr = T.re[k][lane], xi = T.im[k][lane];
        const R xm = sqrt(xr * xr + xi * xi);
        if (xm > R(0)) {
          T.gre[k][lane] += acc * xr / xm;
          T.gim[k][lane] += acc * xi / xm;
        }
      }
      // g_x = IFFT2_unnormalised(g_X) (adjoint of the forward FFT)
      __syncwarp();
      fft_pass<R>(T.gre, T.gim, twi, lane, false);
      __syncwarp();
      if (lane < nw) fft_pass<R>(T.gre, T.gim, twi, lane, true);
      __syncwarp();
      if (lane == 0) {
        ga_acc += static_cast<double>(ga);
        gb_acc += static_cast<double>(gb);
      }
    }
    __syncthreads();
    for (int idx = tid; idx < nw2 * 4; idx += 128) {
      const int pix = idx >> 2, q = idx & 3;
      const int li = pix / nw, lj = pix - li * nw;
      const int c = 4 * g + q;
      C v = mk(tiles[q].gre[li][lj], tiles[q].gim[li][lj]);
      if (c < a.M) {
        const C x = grid[(static_cast<int64_t>(i1 + li) * a.n_j + (j1 + lj)) * a.Mp + c];
        if (isnan(x.x) || isnan(x.y)) v = mk(R(0), R(0));  // NaN inputs enter as constants
      } else {
        v = mk(R(0), R(0));
      }
      wgrad[(wi * nw2 + pix) * a.Mp + 4 * g + q] = v;
    }
  }
  __shared__ double sh_ab[8];
  if (lane == 0) {
    sh_ab[2 * warp] = ga_acc;
    sh_ab[2 * warp + 1] = gb_acc;
  }
  __syncthreads();
  if (tid == 0) {
    b.ab_partial[2 * blockIdx.x] = sh_ab[0] + sh_ab[2] + sh_ab[4] + sh_ab[6];
    b.ab_partial[2 * blockIdx.x + 1] = sh_ab[1] + sh_ab[3] + sh_ab[5] + sh_ab[7];
  }
}

// d L / d alpha and d L / d beta: the per-block partials summed in a fixed order
__global__ void __launch_bounds__(256) k_reduce_ab(const double* __restrict__ part, int n, double* __restrict__ out) {
  __shared__ double sh[2][256];
  const int t = threadIdx.x;
  double a = 0.0, b = 0.0;
  for (int i = t; i < n; i += 256) {
    a += part[2 * i];
    b += part[2 * i + 1];
  }
  sh[0][t] = a;
  sh[1][t] = b;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (t < h) {
      sh[0][t] += sh[0][t + h];
      sh[1][t] += sh[1][t + h];
    }
    __syncthreads();
  }
  if (t == 0) {
    out[0] = sh[0][0];
    out[1] = sh[1][0];
  }
}

cudaError_t launch_reduce_ab(const double* part, int n, double* out, cudaStream_t st) {
  k_reduce_ab<<<1, 256, 0, st>>>(part, n, out);
  return cudaGetLastError();
}

template <typename R>
static size_t clap_bwd_smem() {
  return 4 * sizeof(ClapBwdTile<R>) + 2048 * sizeof(R) + 32 * sizeof(typename CT<R>::C);
}

template <typename R>
static int clap_bwd_blocks(int sm_count) {
  const size_t sm = clap_bwd_smem<R>();
  if (kernel_attributes_once(sm) != cudaSuccess) return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clap_bwd<R>, 128, sm) != cudaSuccess) return 0;
  return sm_count * std::max(per_sm, 1);
}

// Resident blocks of k_clap_bwd on the whole device (the size of the
// alpha/beta partial array); 0 on error.
int clap_bwd_max_blocks(int sm_count, bool fp64) {
  return fp64 ? clap_bwd_blocks<double>(sm_count) : clap_bwd_f32_max_blocks(sm_count);
}

// Launches at most *blocks_out blocks (the partial array's capacity) and
// returns the number launched (0 when there are no windows).
cudaError_t launch_clap_bwd(const ClapBwdArgs& b, bool fp64, const Twiddles32d& td, int* blocks_out,
                            cudaStream_t st) {
  const int64_t ntask = static_cast<int64_t>(b.f.nwi) * b.f.nwj * (b.f.Mp / 4);
  const int64_t blocks = std::min<int64_t>(ntask, static_cast<int64_t>(*blocks_out));
  *blocks_out = static_cast<int>(std::max<int64_t>(blocks, 0));
  if (blocks <= 0) return cudaSuccess;
  if (!fp64) return launch_clap_bwd_f32(b, static_cast<int>(blocks), st);
  k_clap_bwd<double><<<static_cast<unsigned>(blocks), 128, clap_bwd_smem<double>(), st>>>(b, td);
  return cudaGetLastError();
}

// dst[s] = double(src[perm[s]])
__global__ void k_gather_widen(const float* __restrict__ src, double* __restrict__ dst,
                               const int32_t* __restrict__ perm, int64_t n) {
  for (int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < n;
       s += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[s] = static_cast<double>(src[perm[s]]);
}

// dst[perm[s] * words + k] = float(src[s * words + k])
__global__ void k_scatter_narrow(const double* __restrict__ src, float* __restrict__ dst,
                                 const int32_t* __restrict__ perm, int64_t n, int64_t words) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t s = gw; s < n; s += nw) {
    const int64_t r = perm[s];
    for (int64_t k = lane; k < words; k += 32) dst[r * words + k] = static_cast<float>(src[s * words + k]);
  }
}

// dst[perm[s]] = double(src[s]): a per-PS vector back in the caller's row
// order, widened on the device (u8 flags as 0.0 / 1.0)
__device__ __forceinline__ double widen_elem(const float* p, int64_t s) { return static_cast<double>(p[s]); }
__device__ __forceinline__ double widen_elem(const uint8_t* p, int64_t s) { return p[s] ? 1.0 : 0.0; }
template <typename T>
__global__ void k_scatter_widen(const T* __restrict__ src, double* __restrict__ dst, const int32_t* __restrict__ perm,
                                int64_t n) {
  for (int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < n;
       s += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[perm[s]] = widen_elem(src, s);
}

cudaError_t launch_scatter_widen(const void* src, bool flags, double* dst, const int32_t* perm, int64_t n,
                                 cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 255) / 256, 148 * 16);
  if (flags)
    k_scatter_widen<uint8_t><<<static_cast<unsigned>(blocks), 256, 0, st>>>(static_cast<const uint8_t*>(src), dst,
                                                                             perm, n);
  else
    k_scatter_widen<float><<<static_cast<unsigned>(blocks), 256, 0, st>>>(static_cast<const float*>(src), dst, perm,
                                                                           n);
  return cudaGetLastError();
}

cudaError_t launch_gather_widen(const float* src, double* dst, const int32_t* perm, int64_t n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 255) / 256, 148 * 16);
  k_gather_widen<<<static_cast<unsigned>(blocks), 256, 0, st>>>(src, dst, perm, n);
  return cudaGetLastError();
}

cudaError_t launch_scatter_narrow(const double* src, float* dst, const int32_t* perm, int64_t n, int64_t words,
                                  cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 7) / 8, 148 * 16);
  k_scatter_narrow<<<static_cast<unsigned>(blocks), 256, 0, st>>>(src, dst, perm, n, words);
  return cudaGetLastError();
}

// ============================================================== layout ====
// Row gathers/scatters in 4-byte words (row_bytes is a multiple of 4).
__global__ void k_gather_rows(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                              const int32_t* __restrict__ perm, int64_t n, int64_t words, int scatter) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t s = gw; s < n; s += nw) {
    const int64_t r = perm[s];
    const uint32_t* a = scatter ? src + s * words : src + r * words;
    uint32_t* b = scatter ? dst + r * words : dst + s * words;
    for (int64_t k = lane; k < words; k += 32) b[k] = a[k];
  }
}

// one word a row (per-PS vectors): a thread per element, not a warp
__global__ void k_gather_words(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                               const int32_t* __restrict__ perm, int64_t n, int scatter) {
  for (int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < n;
       s += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = perm[s];
    if (scatter)
      dst[r] = src[s];
    else
      dst[s] = src[r];
  }
}

static cudaError_t gather_impl(const void* src, void* dst, const int32_t* perm, int64_t n, int64_t row_bytes,
                               int scatter, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (row_bytes % 4) return cudaErrorInvalidValue;
  if (row_bytes == 4) {
    k_gather_words<<<static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 148 * 8)), 256, 0, st>>>(
        static_cast<const uint32_t*>(src), static_cast<uint32_t*>(dst), perm, n, scatter);
    return cudaGetLastError();
  }
  int64_t blocks = (n + 7) / 8;
  if (blocks > 148 * 16) blocks = 148 * 16;
  k_gather_rows<<<static_cast<unsigned>(blocks), 256, 0, st>>>(static_cast<const uint32_t*>(src),
                                                               static_cast<uint32_t*>(dst), perm, n, row_bytes / 4,
                                                               scatter);
  return cudaGetLastError();
}

cudaError_t launch_gather_rows(const void* src, void* dst, const int32_t* perm, int64_t n, int64_t row_bytes,
                               cudaStream_t st) {
  return gather_impl(src, dst, perm, n, row_bytes, 0, st);
}
cudaError_t launch_scatter_rows(const void* src, void* dst, const int32_t* perm, int64_t n, int64_t row_bytes,
                                cudaStream_t st) {
  return gather_impl(src, dst, perm, n, row_bytes, 1, st);
}

__global__ void k_repad(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t G, int M, int Mp, int eb,
                        int to_padded) {
  const int64_t total = G * static_cast<int64_t>(to_padded ? Mp : M) * eb;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t e = i / eb, byte = i - e * eb;
    if (to_padded) {
      const int64_t g = e / Mp, c = e - g * Mp;
      dst[i] = c < M ? src[(g * M + c) * eb + byte] : 0;
    } else {
      const int64_t g = e / M, c = e - g * M;
      dst[i] = src[(g * Mp + c) * eb + byte];
    }
  }
}

cudaError_t launch_unpad_grid(const void* src, void* dst, int64_t G, int M, int Mp, int eb, cudaStream_t st) {
  k_repad<<<148 * 8, 256, 0, st>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), G, M, Mp, eb, 0);
  return cudaGetLastError();
}
cudaError_t launch_pad_grid(const void* src, void* dst, int64_t G, int M, int Mp, int eb, cudaStream_t st) {
  k_repad<<<148 * 8, 256, 0, st>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), G, M, Mp, eb, 1);
  return cudaGetLastError();
}

template <typename R>
__global__ void k_init_state(const double* __restrict__ w0, const int32_t* __restrict__ perm, int64_t N, R* K, R* w,
                             R* coh) {
  for (int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < N;
       s += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    K[s] = R(0);
    w[s] = static_cast<R>(w0[perm[s]]);
    coh[s] = R(0);
  }
}

cudaError_t launch_init_state(const double* w0, const int32_t* perm, int64_t N, void* K, void* w, void* coh,
                              bool fp64, cudaStream_t st) {
  if (fp64)
    k_init_state<double><<<148 * 4, 256, 0, st>>>(w0, perm, N, static_cast<double*>(K), static_cast<double*>(w),
                                                  static_cast<double*>(coh));
  else
    k_init_state<float><<<148 * 4, 256, 0, st>>>(w0, perm, N, static_cast<float*>(K), static_cast<float*>(w),
                                                 static_cast<float*>(coh));
  return cudaGetLastError();
}

// ph_weight of the last iteration (fill_phase_weight with the K and w that
// iteration used), written in the caller's row order.
template <typename R>
__global__ void k_ph_weight(BinArgs a, const int32_t* __restrict__ perm, int64_t N,
                            typename CT<R>::C* __restrict__ out) {
  using C = typename CT<R>::C;
  const float2* ph = static_cast<const float2*>(a.ph_nm);
  const R* K = static_cast<const R*>(a.K);
  const R* W = static_cast<const R*>(a.w);
  const int64_t total = N * a.M;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t s = i / a.M;
    const int c = static_cast<int>(i - s * a.M);
    const R b = a.bp_row_inv ? static_cast<R>(a.bp[c]) : static_cast<R>(a.bp[i]);
    const R phs = -(b * K[s]);
    R sn, cs;
    sincos_r(phs, &sn, &cs);
    const float2 v = ph[i];
    const C r = cmul_rn(mk(static_cast<R>(v.x), static_cast<R>(v.y)), mk(cs, sn));
    out[static_cast<int64_t>(perm[s]) * a.M + c] = mk(mul_rn(r.x, W[s]), mul_rn(r.y, W[s]));
  }
}

cudaError_t launch_ph_weight(const BinArgs& a, int64_t N, bool fp64, const int32_t* perm, void* out_orig,
                             cudaStream_t st) {
  if (fp64)
    k_ph_weight<double><<<148 * 8, 256, 0, st>>>(a, perm, N, static_cast<double2*>(out_orig));
  else
    k_ph_weight<float><<<148 * 8, 256, 0, st>>>(a, perm, N, static_cast<float2*>(out_orig));
  return cudaGetLastError();
}


// ====================================================== kernel attributes ==
// Every kernel that may take more than 48 KB of dynamic shared memory is opted
// in to the device's per-block maximum once per device and process, before its
// first launch; a launch then only checks its request against that limit.
// Kernel attributes are thereby never changed while another host thread
// captures, instantiates or launches a graph that holds the same kernel
// (contexts run concurrently from several threads).
namespace {
constexpr int kMaxDevices = 64;
std::once_flag g_attr_once[kMaxDevices];
cudaError_t g_attr_result[kMaxDevices];
int g_attr_optin[kMaxDevices];
}  // namespace

cudaError_t kernel_attributes_once(size_t dynamic_smem) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::call_once(g_attr_once[dev], [dev] {
    int optin = 0;
    const cudaError_t r = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const cudaError_t steps[] = {
        r,
        r == cudaSuccess ? clap_f32_attributes(optin) : r,
        r == cudaSuccess ? topofit_f32_attributes(optin) : r,
        r == cudaSuccess ? opt_in_smem(k_clap<double, 4, 0, false>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_clap<double, 4, 24, false>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_clap<double, 4, 0, true>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_clap<double, 4, 24, true>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_topofit_f64<8>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_topofit_f64<16>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_random_hist<4>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_random_hist<8>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_s3_fit, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_topofit_near_max<float>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_topofit_near_max<double>, optin) : r,
        r == cudaSuccess ? opt_in_smem(k_clap_bwd<double>, optin) : r,
    };
    cudaError_t first = cudaSuccess;
    for (const cudaError_t x : steps)
      if (first == cudaSuccess && x != cudaSuccess) first = x;
    g_attr_result[dev] = first;
    g_attr_optin[dev] = optin;
  });
  if (g_attr_result[dev] != cudaSuccess) return g_attr_result[dev];
  return dynamic_smem <= static_cast<size_t>(g_attr_optin[dev]) ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace ps2
