// The FP32 CLAP kernels (clap_f32.cuh): one patch's windows and a batch's.
#include <algorithm>

#include "clap_f32.cuh"

namespace ps2 {

cudaError_t kernel_attributes_once(size_t dynamic_smem);

namespace {

// Row stride of the pyramid-weight table: lane l reads row l, so rows 33 words
// apart put the lanes on different banks.
constexpr int kWtStride = 33;

template <int NW>
struct ClapSmemF {
  ClapTileF<NW == 8 ? 4 : 8> tiles[NW];
  float lp[1024];
  float wt[32 * kWtStride];
};

template <int NW>
__device__ __forceinline__ void clap_consts_f(const ClapArgs& a, ClapSmemF<NW>& m) {
  const int nw2 = a.n_win * a.n_win;
  for (int i = threadIdx.x; i < 1024; i += 32 * NW) m.lp[i] = static_cast<float>(a.low_pass[i]);
  for (int i = threadIdx.x; i < nw2; i += 32 * NW)
    m.wt[(i / a.n_win) * kWtStride + i % a.n_win] = static_cast<float>(a.wscaled[i]);
}

// One window in its tile: on entry the window zero-padded to 32 x 32 (NWIN = 0; a
// compile-time window's padding is never stored), on exit rows and columns < n_win
// hold the filtered values times the pyramid weight / 1024, real parts in im and
// imaginary parts in re.
template <int NWIN, typename Tile>
__device__ __forceinline__ void window_f(Tile& T, const int lane, const ClapArgs& a, const float* lp, const float* wt,
                                         const float (&g)[4], const int rs, const int cs) {
  constexpr int NZ = NWIN > 0 ? NWIN : 32;
  const int nw = NWIN > 0 ? NWIN : a.n_win;
  const float* wrow = wt + (lane - rs) * kWtStride - cs;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
#pragma unroll 1
    for (int p = 2 * half; p < 2 * half + 2; ++p) fft_row<NZ>(T, lane, p, wrow, rs, cs, nw);
    if (half == 0) {
      float o[32];
      smooth_tile(T, lane, g, o);
      float v0, v1;
      median_pair1024(o, &T.hs[0][0], v0, v1);
      gain_tile(T, lane, o, (v0 + v1) * 0.5f, a.alpha_is_one, static_cast<float>(a.alpha), static_cast<float>(a.beta),
                lp);
    }
  }
}

constexpr int kLoadU = 9;  // 16-byte accesses in flight per thread of the window loads

// Window (ix1, ix2) of interferograms NW g .. NW g + NW - 1 through the block's
// tiles: clap_windows' corner (native_stage2.rs:957-995) returned in i1, j1; on
// exit the tiles hold the weighted filtered window.
template <int NW, int NWIN>
__device__ __forceinline__ void compute_f(const ClapArgs& a, const int ix1, const int ix2, const int g,
                                          ClapSmemF<NW>& m, const float (&g7)[4], int& i1, int& j1) {
  constexpr int NT = 32 * NW, NQ = NW / 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  const int n_inc = nw / 4 > 1 ? nw / 4 : 1;
  const float2* __restrict__ grid = static_cast<const float2*>(a.grid);
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
  if (NWIN == 0 && nw < 32) {
    for (int idx = tid; idx < NW * 1024; idx += NT) {
      const int q = idx >> 10, r = (idx >> 5) & 31, c = idx & 31;
      if (r >= nw || c >= nw) m.tiles[q].re[r][c] = m.tiles[q].im[r][c] = 0.f;
    }
  }
  // pixel -> (row, column) by pix * inv_nw >> 16, exact for pix < 1024 and nw <= 32
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  // a thread's pixels are NT / NQ apart: row and column step by step, with one carry
  const int q = (tid % NQ) * 2, c = NW * g + q, pix0 = tid / NQ;
  const int dli = (NT / NQ) / nw, dlj = (NT / NQ) - dli * nw;
  int li = static_cast<int>((static_cast<uint32_t>(pix0) * inv_nw) >> 16), lj = pix0 - li * nw;
  // columns M .. Mp - 1 of the grid are zero, c is even and Mp a multiple of 4
  const float2* src = grid + (static_cast<int64_t>(i1) * a.n_j + j1) * a.Mp + c;
  const int row = a.n_j * a.Mp;  // the window stack, 16 cells or more a grid cell, fits in memory: < 2^31
  const int pix_end = c < a.Mp ? nw2 : 0;
  float* re0 = &m.tiles[q].re[0][0];
  constexpr int kIm = 32 * kTileRow, kNext = sizeof(m.tiles[0]) / sizeof(float);  // tile q's im, tile q + 1
  for (int p0 = pix0; p0 < nw2; p0 += (NT / NQ) * kLoadU) {
    float4 v[kLoadU];
    int at[kLoadU];
#pragma unroll
    for (int u = 0; u < kLoadU; ++u) {
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      at[u] = li * kTileRow + lj;
      // an address per access from li and lj: with one pointer stepped along to the same
      // addresses, the <4, 24, true> instance read other cells (cause not found)
      if (p0 + u * (NT / NQ) < pix_end)
        v[u] = *reinterpret_cast<const float4*>(src + (static_cast<int64_t>(li) * row + lj * a.Mp));
      li += dli;
      lj += dlj;
      if (lj >= nw) {
        lj -= nw;
        ++li;
      }
    }
#pragma unroll
    for (int u = 0; u < kLoadU; ++u) {
      if (p0 + u * (NT / NQ) < nw2) {
        float4 x = v[u];
        if (isnan(x.x) || isnan(x.y)) x.x = x.y = 0.f;  // NaN -> 0 (clap_filter_one_ifg)
        if (isnan(x.z) || isnan(x.w)) x.z = x.w = 0.f;
        re0[at[u]] = x.x;
        re0[at[u] + kIm] = x.y;
        re0[at[u] + kNext] = x.z;
        re0[at[u] + kNext + kIm] = x.w;
      }
    }
  }
  __syncthreads();
  if (NW * g + warp < a.M) {
    window_f<NWIN>(m.tiles[warp], lane, a, m.lp, m.wt, g7, rs, cs);
  } else {
    // an interferogram of the padding: zeros for the window stack
    for (int i = lane; i < nw * nw; i += 32) m.tiles[warp].re[i / nw][i % nw] = m.tiles[warp].im[i / nw][i % nw] = 0.f;
  }
  __syncthreads();
}

template <int NW>
__host__ __device__ __forceinline__ int groups_f(const int Mp) {
  return (Mp + NW - 1) / NW;
}

// One block-task of the window-stack form: window a.w_lo + task / groups.
template <int NW, int NWIN>
__device__ __forceinline__ void task_f(const ClapArgs& a, const int64_t task, ClapSmemF<NW>& m, const float (&g7)[4]) {
  constexpr int NT = 32 * NW, NQ = NW / 2;
  const int groups = groups_f<NW>(a.Mp);
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  // windows number nwi * nwj < 2^31 / 36 cells: 32-bit divisions
  const int w = static_cast<int>(task < INT32_MAX ? static_cast<uint32_t>(task) / static_cast<uint32_t>(groups)
                                                  : task / groups);
  const int g = static_cast<int>(task - static_cast<int64_t>(w) * groups);
  const int64_t wi = a.w_lo + w;
  const int ix1 = static_cast<int>(static_cast<uint32_t>(wi) / static_cast<uint32_t>(a.nwj));
  const int ix2 = static_cast<int>(wi) - ix1 * a.nwj;
  int i1, j1;
  compute_f<NW, NWIN>(a, ix1, ix2, g, m, g7, i1, j1);
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  float2* out = static_cast<float2*>(a.win_out);
  const int q = (threadIdx.x % NQ) * 2, c = NW * g + q, pix0 = threadIdx.x / NQ;
  if (c >= a.Mp) return;
  const int dli = (NT / NQ) / nw, dlj = (NT / NQ) - dli * nw;
  int li = static_cast<int>((static_cast<uint32_t>(pix0) * inv_nw) >> 16), lj = pix0 - li * nw;
  constexpr int kIm = 32 * kTileRow, kNext = sizeof(m.tiles[0]) / sizeof(float);
  const float* re0 = &m.tiles[q].re[0][0];
  float2* dst = out + (wi * nw2 + pix0) * a.Mp + c;
#pragma unroll 3
  for (int pix = pix0; pix < nw2; pix += NT / NQ) {
    const float* s = re0 + li * kTileRow + lj;
    // Mp is a multiple of 4 and c even: c + 1 < Mp, 16-byte aligned
    *reinterpret_cast<float4*>(dst) = make_float4(s[kIm], s[0], s[kNext + kIm], s[kNext]);
    dst += static_cast<int64_t>(NT / NQ) * a.Mp;
    li += dli;
    lj += dlj;
    if (lj >= nw) {
      lj -= nw;
      ++li;
    }
  }
}

// The weighted window added to (or, for a cell no earlier window of the block
// covered, stored in) the block's partial sums: see clap_accum_tiles.
constexpr int kAccU = 6;
template <int NW>
__device__ __forceinline__ void accum_f(const ClapArgs& a, const ClapSmemF<NW>& m, double2* __restrict__ part,
                                           const int64_t blk, const int box, const int i1, const int j1, const int r0,
                                           const int c0, const int pi1, const int pj1, const int g, const int nw,
                                           const int nw2, const uint32_t inv_nw) {
  constexpr int NT = 32 * NW, NI = NW;
  const int n_items = nw2 * NI;
  for (int b0 = threadIdx.x; b0 < n_items; b0 += NT * kAccU) {
    double2 old[kAccU];
    int64_t off[kAccU];
    int li[kAccU], lj[kAccU], qq[kAccU];
    bool live[kAccU], first[kAccU];
#pragma unroll
    for (int u = 0; u < kAccU; ++u) {
      const int idx = b0 + u * NT;
      const int pix = idx / NI, q = idx % NI, c = NI * g + q;
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
    for (int u = 0; u < kAccU; ++u) {
      if (!live[u]) continue;
      const double vx = static_cast<double>(m.tiles[qq[u]].im[li[u]][lj[u]]);
      const double vy = static_cast<double>(m.tiles[qq[u]].re[li[u]][lj[u]]);
      part[off[u]] = first[u] ? make_double2(vx, vy) : make_double2(__dadd_rn(old[u].x, vx), __dadd_rn(old[u].y, vy));
    }
  }
}

// One block-task of the fused form: window block a.w_lo + task / groups.
template <int NW, int NWIN>
__device__ __forceinline__ void block_task_f(const ClapArgs& a, const int64_t task, ClapSmemF<NW>& m,
                                                const float (&g7)[4]) {
  const int groups = groups_f<NW>(a.Mp);
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  const int n_inc = nw / 4 > 1 ? nw / 4 : 1;
  const int box = clap_box(nw);
  const int nbj = clap_block_rows(a.nwj);
  const int64_t blk = a.w_lo + task / groups;
  const int g = static_cast<int>(task - (blk - a.w_lo) * groups);
  const int bi = static_cast<int>(blk / nbj), bj = static_cast<int>(blk - static_cast<int64_t>(bi) * nbj);
  const int ixa = kClapBlockWin * bi, ixb = min(ixa + kClapBlockWin, a.nwi);
  const int jxa = kClapBlockWin * bj, jxb = min(jxa + kClapBlockWin, a.nwj);
  const int r0 = min(ixa * n_inc, a.n_i - nw), c0 = min(jxa * n_inc, a.n_j - nw);
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  constexpr int kNone = -(1 << 20);
  for (int ix1 = ixa; ix1 < ixb; ++ix1) {
    const int pi1 = ix1 > ixa ? min((ix1 - 1) * n_inc, a.n_i - nw) : kNone;
    for (int ix2 = jxa; ix2 < jxb; ++ix2) {
      const int pj1 = ix2 > jxa ? min((ix2 - 1) * n_inc, a.n_j - nw) : kNone;
      int i1, j1;
      compute_f<NW, NWIN>(a, ix1, ix2, g, m, g7, i1, j1);
      accum_f<NW>(a, m, static_cast<double2*>(a.part), blk, box, i1, j1, r0, c0, pi1, pj1, g, nw, nw2, inv_nw);
    }
  }
}

__device__ __forceinline__ void taps_f(const ClapArgs& a, float (&g)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) g[i] = static_cast<float>(a.g7[i]);  // symmetric: taps 0..3
}

// FUSED: window blocks into the partials; otherwise windows into the window
// stack. Sixteen warps an SM in two blocks of eight (shared memory and 128
// registers allow no more). 256 x 256 cells x 150 ifg: 2.57 -> 1.85 ms a launch (4,850 instructions a
// window and interferogram against 6,800).
template <int NW, int NWIN, bool FUSED>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? 2 : 3) k_clap_f32(ClapArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ClapSmemF<NW>& m = *reinterpret_cast<ClapSmemF<NW>*>(smem_raw);
  clap_consts_f<NW>(a, m);
  float g7[4];
  taps_f(a, g7);
  const int64_t nunit = a.w_n > 0 ? a.w_n
                        : FUSED ? static_cast<int64_t>(clap_block_rows(a.nwi)) * clap_block_rows(a.nwj)
                                : static_cast<int64_t>(a.nwi) * a.nwj;
  const int64_t ntask = nunit * groups_f<NW>(a.Mp);
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    if constexpr (FUSED)
      block_task_f<NW, NWIN>(a, task, m, g7);
    else
      task_f<NW, NWIN>(a, task, m, g7);
  }
}

// Block-tasks numbered patch after patch; the per-patch constants are reloaded
// where a block's tasks change patch. NWIN = 24 when every patch has that window.
template <int NWIN>
__global__ void __launch_bounds__(256, 2) k_batch_clap(BatchArgs b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ClapSmemF<8>& m = *reinterpret_cast<ClapSmemF<8>*>(smem_raw);
  float g7[4];
  int cur = -1;
  const int64_t total = b.clap_prefix[b.P];
  for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
    const int p = find_patch(b.clap_prefix, b.P, u);
    if (!b.active[p]) continue;
    const ClapArgs& a = b.patch[p].clap;
    if (p != cur) {
      // the previous task's readers of lp / wt passed its last barrier
      clap_consts_f<8>(a, m);
      taps_f(a, g7);
      cur = p;
    }
    if (a.part)
      block_task_f<8, NWIN>(a, u - b.clap_prefix[p], m, g7);
    else
      task_f<8, NWIN>(a, u - b.clap_prefix[p], m, g7);
  }
}

// ---- stage 3: the filtered value of a 32 x 32 patch at one cell ----------------
// A block's four patches of one job (PS cell): interferograms 4 g .. 4 g + 3. Four
// blocks an SM (57 KB and 128 registers each), sixteen warps as with eight a block,
// and at most three idle warps at the end of the interferograms. 16,384 cells x 60
// ifg: 10.9 -> 6.7 ms, with the window kernel's passes, inlined here (no spills at 128
// registers; 7.3 ms with the transform out of line).
struct S3Smem {
  ClapTileF<8> tiles[4];
  float lp[1024];
  float2 wp[32];  // e^{+2 pi i k / 32}
};

// The patch in its tile -> the filtered value at (bi, bj), times 1024: the inverse
// transform evaluated at that one point,
// y = sum_{k1,k2} Y[k1][k2] e^{+2 pi i (k1 bi + k2 bj) / 32}.
template <typename Tile>
__device__ __forceinline__ float2 s3_patch_point(Tile& T, const int lane, const S3ClapArgs& a, const S3Smem& m,
                                                 const float (&g)[4], const int bi, const int bj) {
#pragma unroll 1
  for (int p = kForward1; p <= kForward2; ++p) fft_row_inline<32, 1>(T, lane, p, nullptr, 0, 0, 32);
  float o[32];
  smooth_tile(T, lane, g, o);
  float v0, v1;
  median_pair1024(o, &T.hs[0][0], v0, v1);
  gain_tile(T, lane, o, (v0 + v1) * 0.5f, a.alpha_is_one, static_cast<float>(a.alpha), static_cast<float>(a.beta),
            m.lp);
  // the lane's column of the spectrum lies in its row of the tile
  float ax = 0.f, ay = 0.f;
#pragma unroll
  for (int k = 0; k < 32; k += 2) {
    const float2 g2 = *reinterpret_cast<const float2*>(&T.hs[lane][k]);
    const float2 yr = __fmul2_rn(*reinterpret_cast<const float2*>(&T.re[lane][k]), g2);
    const float2 yi = __fmul2_rn(*reinterpret_cast<const float2*>(&T.im[lane][k]), g2);
    const float2 w0 = m.wp[(k * bi) & 31], w1 = m.wp[((k + 1) * bi) & 31];
    ax = __fadd_rn(ax, __fmaf_rn(yr.x, w0.x, -__fmul_rn(yi.x, w0.y)));
    ay = __fadd_rn(ay, __fmaf_rn(yr.x, w0.y, __fmul_rn(yi.x, w0.x)));
    ax = __fadd_rn(ax, __fmaf_rn(yr.y, w1.x, -__fmul_rn(yi.y, w1.y)));
    ay = __fadd_rn(ay, __fmaf_rn(yr.y, w1.y, __fmul_rn(yi.y, w1.x)));
  }
  const float2 w = m.wp[(lane * bj) & 31];
  return make_float2(warp_sum(__fmaf_rn(ax, w.x, -__fmul_rn(ay, w.y))),
                     warp_sum(__fmaf_rn(ay, w.x, __fmul_rn(ax, w.y))));
}

// VEC: an even row stride of the grid, so an even interferogram and its neighbour
// come in one 16-byte access (the columns past M up to the stride are zero).
template <bool VEC>
__global__ void __launch_bounds__(128, 4) k_s3_clap(S3ClapArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S3Smem& m = *reinterpret_cast<S3Smem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < 1024; i += 128) m.lp[i] = static_cast<float>(a.low_pass[i]);
  if (tid < 16) {
    const float c = tid == 8 ? a.quarter_cos : kCos32[tid];
    m.wp[tid] = make_float2(c, kSin32[tid]);
    m.wp[tid + 16] = make_float2(-c, -kSin32[tid]);
  }
  float g7[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) g7[i] = static_cast<float>(a.g7[i]);
  const int M = a.M;
  const int64_t ntask = a.n_jobs * a.ngroups;
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    const int64_t job = task < INT32_MAX ? static_cast<uint32_t>(task) / static_cast<uint32_t>(a.ngroups)
                                         : task / a.ngroups;
    const int g = static_cast<int>(task - job * a.ngroups);
    const int4 jb = *reinterpret_cast<const int4*>(a.jobs + 4 * job);
    const int i0 = jb.x, j0 = jb.y, bi = jb.z, bj = jb.w;
    const int c_warp = 4 * g + warp;
    if (i0 < 0) {
      // the 32-cell patch does not fit: the reference sets ph_patch2 to 0
      if (lane == 0 && c_warp < M) a.job_out[job * M + c_warp] = make_float2(0.f, 0.f);
      continue;
    }
    __syncthreads();
    constexpr int U = 8, QN = VEC ? 2 : 4, STEP = 128 / QN;  // pixels a round
    const int q = (tid % QN) * (VEC ? 2 : 1), c = 4 * g + q, pix0 = tid / QN;
    // a thread's pixels: STEP apart, whole rows of 32
    const float2* src = a.grid + (static_cast<int64_t>(i0 + (pix0 >> 5)) * a.grid_cols + (j0 + (pix0 & 31))) * a.grid_stride + c;
    const int64_t step = static_cast<int64_t>(STEP / 32) * a.grid_cols * a.grid_stride;
    for (int p0 = pix0; p0 < 1024; p0 += STEP * U) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
          if (c < a.grid_stride) v[u] = *reinterpret_cast<const float4*>(src);
        } else if (c < M) {
          const float2 x = *src;
          v[u].x = x.x;
          v[u].y = x.y;
        }
        src += step;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int pix = p0 + u * STEP, li = pix >> 5, lj = pix & 31;
        float4 x = v[u];
        if (isnan(x.x) || isnan(x.y)) x.x = x.y = 0.f;
        if (isnan(x.z) || isnan(x.w)) x.z = x.w = 0.f;
        const bool own = li == bi && lj == bj;
        const bool osf = c == 0 && abs(li - bi) <= a.slc_rad && abs(lj - bj) <= a.slc_rad;
        if (own || osf) x.x = x.y = 0.f;
        if (own) x.z = x.w = 0.f;
        m.tiles[q].re[li][lj] = x.x;
        m.tiles[q].im[li][lj] = x.y;
        if (VEC) {
          m.tiles[q + 1].re[li][lj] = x.z;
          m.tiles[q + 1].im[li][lj] = x.w;
        }
      }
    }
    __syncthreads();
    if (c_warp < M) {
      const float2 r = s3_patch_point(m.tiles[warp], lane, a, m, g7, bi, bj);
      if (lane == 0) a.job_out[job * M + c_warp] = make_float2(r.x * (1.f / 1024.f), r.y * (1.f / 1024.f));
    }
  }
}

// ---- adjoint of a window -------------------------------------------------------
// Per warp: the window (x) and the weighted gradient of its output (gy), both
// transformed by the passes of the forward kernel; the spectrum X, its smoothed
// magnitude and median are recomputed, not stored. On exit the tile `G` holds the
// gradient of x with re and im exchanged. 96 KB a block of four warps, two an SM.
// 96 x 96 cells x 40 ifg: 457 -> 335 us.
struct AdjTile {
  float re[32][kTileRow], im[32][kTileRow], hs[32][kTileRow];
  struct Grad {
    float re[32][kTileRow], im[32][kTileRow];
  } G;
  float pad[8];
};
struct AdjSmem {
  AdjTile tiles[4];
  float lp[1024];
  float wt[32 * kWtStride];
};

template <int NZ>
__device__ __forceinline__ void adjoint_window(AdjTile& T, const int lane, const ClapArgs& a, const float* lp,
                                               const float (&g)[4], double& ga_acc, double& gb_acc) {
  fft_row<NZ, 1>(T, lane, kForward1, nullptr, 0, 0, NZ);
  fft_row<NZ, 2>(T.G, lane, kForward1, nullptr, 0, 0, NZ);
  fft_row<NZ, 1>(T, lane, kForward2, nullptr, 0, 0, NZ);
  fft_row<NZ, 2>(T.G, lane, kForward2Plain, nullptr, 0, 0, NZ);
  const float alpha = static_cast<float>(a.alpha), beta = static_cast<float>(a.beta);
  float o[32], t[32];
  smooth_tile(T, lane, g, o);
  float v0, v1;
  median_pair1024(o, &T.hs[0][0], v0, v1);
  const float med = (v0 + v1) * 0.5f;
  const float inv_med = med != 0.f ? 1.f / med : 1.f;
  float gmed = 0.f, ga = 0.f, gb = 0.f;
  // t: dL/d(smoothed |X|), starting with the direct term; G becomes g_X from Y = X G
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const float xr = T.re[lane][k], xi = T.im[lane][k], gyr = T.G.re[lane][k], gyi = T.G.im[lane][k];
    const float hn = o[k] * inv_med;
    const float pw = a.alpha_is_one ? hn : powf(hn, alpha);
    const bool act = pw - 1.f > 0.f;
    const float gain = (act ? pw - 1.f : 0.f) * beta + lp[k * 32 + lane];
    const float gG = xr * gyr + xi * gyi;
    float ghn = 0.f;
    if (act) {
      ghn = gG * beta * (a.alpha_is_one ? 1.f : alpha * powf(hn, alpha - 1.f));
      gb += gG * (pw - 1.f);
      ga += gG * beta * pw * logf(hn);
    }
    if (med != 0.f) gmed += ghn * (-o[k] * inv_med * inv_med);
    t[k] = med != 0.f ? ghn * inv_med : ghn;
    T.G.re[lane][k] = gyr * gain;
    T.G.im[lane][k] = gyi * gain;
  }
  gmed = warp_sum(gmed);
  ga = warp_sum(ga);
  gb = warp_sum(gb);
  if (med != 0.f) {
    // med = (v0 + v1) / 2 of the smoothed magnitudes; ties share evenly
    unsigned cnt = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) cnt += (o[k] == v0 ? 1u : 0u) + (o[k] == v1 ? 0x10000u : 0u);
    cnt = __reduce_add_sync(kFull, cnt);
    const float c0 = static_cast<float>(cnt & 0xffffu), c1 = static_cast<float>(cnt >> 16);
    const float share0 = v0 == v1 ? gmed / c0 : 0.5f * gmed / c0;
    const float share1 = v0 == v1 ? 0.f : 0.5f * gmed / c1;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      if (o[k] == v0)
        t[k] += share0;
      else if (o[k] == v1)
        t[k] += share1;
    }
  }
  // adjoint of the separable smoothing: along the lane's column, then along the rows
  smooth32(t, g, o);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 32; ++k) T.hs[k][lane] = o[k];
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 32; ++c) t[c] = T.hs[lane][c];
  smooth32(t, g, o);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 32; ++c) T.hs[c][lane] = o[c];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    // H = |X|:  g_X += g_H X / |X|
    const float xr = T.re[lane][k], xi = T.im[lane][k];
    const float xm = sqrt_rn(xr * xr + xi * xi);
    const float q = xm > 0.f ? T.hs[lane][k] / xm : 0.f;
    T.G.re[lane][k] += q * xr;
    T.G.im[lane][k] += q * xi;
  }
  // g_x = the unnormalised inverse transform of g_X (adjoint of the forward one)
  fft_row<NZ, 2>(T.G, lane, kInverse1Plain, nullptr, 0, 0, NZ);
  fft_row<NZ, 2>(T.G, lane, kInverse2Plain, nullptr, 0, 0, NZ);
  if (lane == 0) {
    ga_acc += static_cast<double>(ga);
    gb_acc += static_cast<double>(gb);
  }
}

template <int NWIN>
__global__ void __launch_bounds__(128, 2) k_clap_bwd_f32(ClapBwdArgs b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  AdjSmem& m = *reinterpret_cast<AdjSmem*>(smem_raw);
  const ClapArgs& a = b.f;
  constexpr int NZ = NWIN > 0 ? NWIN : 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nw = NWIN > 0 ? NWIN : a.n_win, nw2 = nw * nw;
  for (int i = tid; i < 1024; i += 128) m.lp[i] = static_cast<float>(a.low_pass[i]);
  for (int i = tid; i < nw2; i += 128) m.wt[(i / nw) * kWtStride + i % nw] = static_cast<float>(a.wscaled[i]);
  float g7[4];
  taps_f(a, g7);
  const int n_inc = nw / 4 > 1 ? nw / 4 : 1;
  const uint32_t ngroups = static_cast<uint32_t>(a.Mp / 4);
  const int64_t ntask = static_cast<int64_t>(a.nwi) * a.nwj * ngroups;
  const uint32_t inv_nw = (65536u + static_cast<uint32_t>(nw) - 1u) / static_cast<uint32_t>(nw);
  const float2* __restrict__ grid = static_cast<const float2*>(a.grid);
  const float2* __restrict__ gfilt = static_cast<const float2*>(b.gfilt);
  float2* __restrict__ wgrad = static_cast<float2*>(b.wgrad);
  double ga_acc = 0.0, gb_acc = 0.0;
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    const int wi = static_cast<int>(task < INT32_MAX ? static_cast<uint32_t>(task) / ngroups : task / ngroups);
    const int g = static_cast<int>(task - static_cast<int64_t>(wi) * ngroups);
    const int ix1 = wi / a.nwj, ix2 = wi - ix1 * a.nwj;
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
    if (NWIN == 0 && nw < 32) {
      for (int idx = tid; idx < 4 * 1024; idx += 128) {
        const int q = idx >> 10, r = (idx >> 5) & 31, c = idx & 31;
        if (r >= nw || c >= nw)
          m.tiles[q].re[r][c] = m.tiles[q].im[r][c] = m.tiles[q].G.re[r][c] = m.tiles[q].G.im[r][c] = 0.f;
      }
    }
    // two interferograms (16 bytes) of the window and of the gradient per access;
    // columns M .. Mp - 1 of both grids are zero
    const int q = (tid & 1) * 2, c = 4 * g + q;
    for (int pix = tid >> 1; pix < nw2; pix += 64) {
      const int li = static_cast<int>((static_cast<uint32_t>(pix) * inv_nw) >> 16), lj = pix - li * nw;
      const int64_t at = (static_cast<int64_t>(i1 + li) * a.n_j + (j1 + lj)) * a.Mp + c;
      float4 v = *reinterpret_cast<const float4*>(grid + at);
      const float4 go = *reinterpret_cast<const float4*>(gfilt + at);
      if (isnan(v.x) || isnan(v.y)) v.x = v.y = 0.f;
      if (isnan(v.z) || isnan(v.w)) v.z = v.w = 0.f;
      const float wv = (li < rs || lj < cs) ? 0.f : m.wt[(li - rs) * kWtStride + (lj - cs)];
      // out += w y  =>  g_y = w g_out
      m.tiles[q].re[li][lj] = v.x;
      m.tiles[q].im[li][lj] = v.y;
      m.tiles[q].G.re[li][lj] = go.x * wv;
      m.tiles[q].G.im[li][lj] = go.y * wv;
      m.tiles[q + 1].re[li][lj] = v.z;
      m.tiles[q + 1].im[li][lj] = v.w;
      m.tiles[q + 1].G.re[li][lj] = go.z * wv;
      m.tiles[q + 1].G.im[li][lj] = go.w * wv;
    }
    __syncthreads();
    if (4 * g + warp < a.M) adjoint_window<NZ>(m.tiles[warp], lane, a, m.lp, g7, ga_acc, gb_acc);
    __syncthreads();
    for (int pix = tid >> 1; pix < nw2; pix += 64) {
      const int li = static_cast<int>((static_cast<uint32_t>(pix) * inv_nw) >> 16), lj = pix - li * nw;
      const float4 x =
          *reinterpret_cast<const float4*>(grid + (static_cast<int64_t>(i1 + li) * a.n_j + (j1 + lj)) * a.Mp + c);
      float4 v = make_float4(m.tiles[q].G.im[li][lj], m.tiles[q].G.re[li][lj], m.tiles[q + 1].G.im[li][lj],
                             m.tiles[q + 1].G.re[li][lj]);
      // NaN inputs enter as constants; columns past M have no gradient
      if (c >= a.M || isnan(x.x) || isnan(x.y)) v.x = v.y = 0.f;
      if (c + 1 >= a.M || isnan(x.z) || isnan(x.w)) v.z = v.w = 0.f;
      *reinterpret_cast<float4*>(wgrad + (static_cast<int64_t>(wi) * nw2 + pix) * a.Mp + c) = v;
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

template <int NW, int NWIN, bool FUSED>
cudaError_t launch_form(const ClapArgs& a, const int64_t ntask, int sm_count, cudaStream_t st) {
  const size_t sm = sizeof(ClapSmemF<NW>);
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clap_f32<NW, NWIN, FUSED>, 32 * NW, sm);
  if (e != cudaSuccess) return e;
  if (a.blocks_per_sm > 0 && a.blocks_per_sm < per_sm) per_sm = a.blocks_per_sm;
  const int64_t blocks = std::min<int64_t>(ntask, static_cast<int64_t>(sm_count) * (per_sm > 0 ? per_sm : 1));
  k_clap_f32<NW, NWIN, FUSED><<<static_cast<unsigned>(blocks), 32 * NW, sm, st>>>(a);
  return cudaGetLastError();
}

// Windows, or window blocks where the partials are asked for, of a launch.
int64_t units_f(const ClapArgs& a) {
  if (a.w_n > 0) return a.w_n;
  return a.part ? static_cast<int64_t>(clap_block_rows(a.nwi)) * clap_block_rows(a.nwj)
                : static_cast<int64_t>(a.nwi) * a.nwj;
}

template <int NW>
cudaError_t launch_nw(const ClapArgs& a, int sm_count, cudaStream_t st) {
  if (a.nwi <= 0 || a.nwj <= 0) return cudaSuccess;
  const int64_t ntask = units_f(a) * groups_f<NW>(a.Mp);
  if (ntask <= 0) return cudaSuccess;
  if (a.n_win == 24)
    return a.part ? launch_form<NW, 24, true>(a, ntask, sm_count, st)
                  : launch_form<NW, 24, false>(a, ntask, sm_count, st);
  return a.part ? launch_form<NW, 0, true>(a, ntask, sm_count, st)
                : launch_form<NW, 0, false>(a, ntask, sm_count, st);
}

}  // namespace

int64_t batch_clap_groups(int Mp) { return groups_f<8>(Mp); }

// Warps a block unless the caller says. 8 (two blocks, sixteen warps an SM) hide more
// than 4 (three blocks, twelve), and 4 finish a partly filled device sooner: 4 where
// all their blocks fit at once, else 8 where those do, else by the padding: with Mp mod
// 8 = 4 blocks of 8 idle 4 / (Mp + 4) of their warps, which costs more than 12 for 16
// up to Mp = 60, and at any Mp where two rounds of blocks do or in window blocks, whose
// few long tasks leave a longer tail. us with 4 | 8 warps, window stack: 200 x 200 cells
// 12 ifg 123 | 155, 28 278 | 294, 60 567 | 565, 100 932 | 887, 148 1369 | 1318, 150
// 1422 | 1328; 64 x 64 x 28 38.0 | 33.6; 40 x 40 cells 100 ifg 31.7 | 33.7, 116 38.5 |
// 33.9, 148 42.0 | 44.5. Window blocks: 40 x 40 x 150 180 | 240; 128 x 128 x 132 531 |
// 655, 76 385 | 372; 200 x 200 x 84 871 | 954.
cudaError_t launch_clap_f32(const ClapArgs& a, int sm_count, cudaStream_t st) {
  int nw = a.nw_block;
  if (nw != 4 && nw != 8) {
    const int64_t units = units_f(a), fours = units * groups_f<4>(a.Mp), once = static_cast<int64_t>(sm_count) * 3;
    if (fours <= once)
      nw = 4;
    else if (!a.part && units * groups_f<8>(a.Mp) <= static_cast<int64_t>(sm_count) * 2)
      nw = 8;
    else
      nw = a.Mp % 8 == 4 && (a.part || a.Mp <= 60 || fours <= 2 * once) ? 4 : 8;
  }
  return nw == 4 ? launch_nw<4>(a, sm_count, st) : launch_nw<8>(a, sm_count, st);
}

cudaError_t launch_batch_clap(const BatchArgs& b, int64_t total, bool win24, int sm_count, cudaStream_t st) {
  if (total <= 0) return cudaSuccess;
  const size_t sm = sizeof(ClapSmemF<8>);
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min<int64_t>(total, static_cast<int64_t>(sm_count) * 2);
  if (win24)
    k_batch_clap<24><<<static_cast<unsigned>(blocks), 256, sm, st>>>(b);
  else
    k_batch_clap<0><<<static_cast<unsigned>(blocks), 256, sm, st>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_s3_clap(const S3ClapArgs& a, int sm_count, cudaStream_t st) {
  const int64_t ntask = a.n_jobs * a.ngroups;
  if (ntask <= 0) return cudaSuccess;
  const size_t sm = sizeof(S3Smem);
  cudaError_t e = kernel_attributes_once(sm);
  if (e != cudaSuccess) return e;
  const unsigned blocks = static_cast<unsigned>(std::min<int64_t>(ntask, static_cast<int64_t>(sm_count) * 4));
  if (a.grid_stride % 2 == 0)
    k_s3_clap<true><<<blocks, 128, sm, st>>>(a);
  else
    k_s3_clap<false><<<blocks, 128, sm, st>>>(a);
  return cudaGetLastError();
}

int clap_bwd_f32_max_blocks(int sm_count) {
  const size_t sm = sizeof(AdjSmem);
  if (kernel_attributes_once(sm) != cudaSuccess) return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_clap_bwd_f32<24>, 128, sm) != cudaSuccess) return 0;
  return sm_count * std::max(per_sm, 1);
}

cudaError_t launch_clap_bwd_f32(const ClapBwdArgs& b, int blocks, cudaStream_t st) {
  if (b.f.n_win == 24)
    k_clap_bwd_f32<24><<<static_cast<unsigned>(blocks), 128, sizeof(AdjSmem), st>>>(b);
  else
    k_clap_bwd_f32<0><<<static_cast<unsigned>(blocks), 128, sizeof(AdjSmem), st>>>(b);
  return cudaGetLastError();
}

cudaError_t clap_f32_attributes(int optin) {
  const cudaError_t steps[] = {
      opt_in_smem(k_clap_f32<4, 24, false>, optin), opt_in_smem(k_clap_f32<4, 24, true>, optin),
      opt_in_smem(k_clap_f32<4, 0, false>, optin),  opt_in_smem(k_clap_f32<4, 0, true>, optin),
      opt_in_smem(k_clap_f32<8, 24, false>, optin), opt_in_smem(k_clap_f32<8, 24, true>, optin),
      opt_in_smem(k_clap_f32<8, 0, false>, optin),  opt_in_smem(k_clap_f32<8, 0, true>, optin),
      opt_in_smem(k_batch_clap<24>, optin),         opt_in_smem(k_batch_clap<0>, optin),
      opt_in_smem(k_s3_clap<true>, optin),          opt_in_smem(k_s3_clap<false>, optin),
      opt_in_smem(k_clap_bwd_f32<24>, optin),       opt_in_smem(k_clap_bwd_f32<0>, optin),
  };
  for (const cudaError_t x : steps)
    if (x != cudaSuccess) return x;
  return cudaSuccess;
}

}  // namespace ps2
