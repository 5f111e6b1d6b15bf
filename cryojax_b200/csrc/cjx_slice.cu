// Forward Fourier-slice + CTF kernels (sm_100a).
//
// Resize path ((Py, Px) != (N, N)), three passes per chunk of images, with
// the two intermediates kept in a workspace sized so a chunk stays L2
// resident:
//   A  gather + column inverse FFT: one warp per slice column kx.  The warp
//      samples the N points of that column of the rotated central plane,
//      makes columns kx = 0 and kx = N/2 Hermitian in ky (the irfftn of the
//      reference ignores the non-Hermitian part there), runs an N-point
//      inverse FFT and keeps the Py rows of the real-space crop/pad window.
//   B  rows: two rows packed as A + iB, Hermitian-extended, N-point inverse
//      FFT (= irfft of both rows), crop/pad window to Px, Px-point forward
//      FFT, split into the two rfft half rows.
//   C  columns: Py-point forward FFT of each half-plane column, then scale,
//      CTF, envelope and translation, written to the output.
// No-resize path ((Py, Px) == (N, N)): one fused kernel samples each output
// pixel and applies the epilogue directly.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>
#include <cmath>

#include "cjx_common.cuh"
#include "cjx_profile.cuh"

namespace cjx {

// ---------------------------------------------------------------------------
// Pass A
// ---------------------------------------------------------------------------
template <int S, typename Layout, bool PRIMES>
__global__ void __launch_bounds__(kWarps * 32)
    k_gather_colifft(const float2* __restrict__ grid, const cjx_image_params* __restrict__ params,
                     const int32_t* __restrict__ order, float2* __restrict__ t1, const __grid_constant__ SliceGeom g, int64_t k0) {
  const Layout L(g.n);
  extern __shared__ float2 smem[];
  const int n = g.n, h = n / 2;
  const int stride = 2 * n + 2;  // per-warp buffers (+2 to stagger banks)
  float2* tw = smem;
  float2* bufs = smem + n;
  build_twiddles(tw, n);

  const int64_t k = k0 + blockIdx.y;
  const int64_t img = order ? (int64_t)order[k] : k;
  const double* R = params[img].rot;
  const float r00 = (float)R[0], r01 = (float)R[1];
  const float r10 = (float)R[3], r11 = (float)R[4];
  const float r20 = (float)R[6], r21 = (float)R[7];
  const bool wrap = !(g.flags & CJX_ZERO_FILL_NEGATIVE);
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j0 = blockIdx.x * kWarps;
  const int j = j0 + warp;
  float2* a = bufs + warp * stride;
  float2* b = a + n;
  if (j < g.nxh) {
    const float ux = (float)fft_index(j, n);
    const float bx = r00 * ux, by = r10 * ux, bz = r20 * ux;
    for (int i0 = lane; i0 < n; i0 += 32 * S) {
      float ox[S], oy[S], oz[S];
      bool act[S];
      float2 val[S];
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int i = i0 + 32 * s;
        act[s] = i < n;
        const float vy = (float)fft_index(act[s] ? i : 0, n);
        ox[s] = fmaf(r01, vy, bx);
        oy[s] = fmaf(r11, vy, by);
        oz[s] = fmaf(r21, vy, bz);
      }
      gather_samples<S>(grid, n, L, ox, oy, oz, act, wrap, g.fill, val);
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (act[s]) a[i0 + 32 * s] = val[s];
    }
    __syncwarp();
    if (j == 0 || ((n % 2 == 0) && j == h)) {
      // S'[v] = (S[v] + conj(S[-v])) / 2  (covers the mode="real" fix at v = 0, N/2)
      for (int i = lane; i <= n / 2; i += 32) {
        const int i2 = (i == 0) ? 0 : n - i;
        const float2 x = a[i], y = a[i2];
        const float2 sv = make_float2(0.5f * (x.x + y.x), 0.5f * (x.y - y.y));
        a[i] = sv;
        a[i2] = cconj(sv);
      }
      __syncwarp();
    }
    warp_fft<+1, PRIMES>(a, b, g.plan_n, tw, lane);
  }
  __syncthreads();

  // The FFT result sits in buffer a after an even number of Stockham stages,
  // in b after an odd number (or after the direct DFT).
  const int res_off = (g.plan_n.nstages == 0 || (g.plan_n.nstages & 1)) ? n : 0;
  const int ncols = min(kWarps, g.nxh - j0);
  float2* dst = t1 + (size_t)blockIdx.y * g.py * g.ld1 + j0;
  for (int e = threadIdx.x; e < g.py * kWarps; e += blockDim.x) {
    const int m = e / kWarps, jj = e % kWarps;
    if (jj < ncols) {
      const int src = win_src(m, n, g.py, g.pad_left_y);
      dst[(size_t)m * g.ld1 + jj] = (src >= 0) ? bufs[jj * stride + res_off + src] : make_float2(0.f, 0.f);
    }
  }
}

// ---------------------------------------------------------------------------
// Pass A, split form: a shared-memory-free gather kernel (the L1 cache keeps
// its full capacity for the corner loads of neighbouring samples) writing the
// half-plane slice H[kx][ky] to an L2-resident buffer, then a column kernel
// that runs the Hermitian fix, inverse FFT and window on H.
// ---------------------------------------------------------------------------
// Resident CTAs per SM that the split gather must allow for (register cap).
// Trilinear instances of one or two samples per lane: 4 (64 registers; at the
// 71 that the compiler takes without the cap, 3 fit and N = 360 took 0.40 ms per
// 512 images instead of 0.35).  Spline instances: 64 taps per sample would take
// about 170 registers if every load were hoisted; 2 CTAs cap them at 128.
template <int S, typename Layout>
constexpr int kGatherCtas = is_spline_layout<Layout>::value ? 2 : (S <= 2 ? 4 : 1);

template <int S, typename Layout, int MAP>
__global__ void __launch_bounds__(256, (kGatherCtas<S, Layout>))
    k_gather_slice(const float2* __restrict__ grid, const cjx_image_params* __restrict__ params,
                   const int32_t* __restrict__ order, float2* __restrict__ hbuf, SliceGeom g, int64_t k0) {
  const Layout L(g.n);
  const int n = g.n;
  const int64_t k = k0 + blockIdx.z;
  const int64_t img = order ? (int64_t)order[k] : k;
  const double* R = params[img].rot;
  const float r00 = (float)R[0], r01 = (float)R[1];
  const float r10 = (float)R[3], r11 = (float)R[4];
  const float r20 = (float)R[6], r21 = (float)R[7];
  const bool wrap = !(g.flags & CJX_ZERO_FILL_NEGATIVE);
  // CTA patch: 16 columns x 16*S rows, S sample rows 16 apart per thread
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int du, dv;
  gather_lane_offsets<MAP>(warp, lane, du, dv);
  const int u = blockIdx.x * 16 + du;
  if (u >= g.ncols) return;
  const int vbase = blockIdx.y * (16 * S) + dv;
  const float ux = (float)fft_index(u, n);
  const float bx = r00 * ux, by = r10 * ux, bz = r20 * ux;
  float ox[S], oy[S], oz[S];
  bool act[S];
  float2 val[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int v = vbase + 16 * s;
    act[s] = v < n;
    const float vy = (float)fft_index(act[s] ? v : 0, n);
    ox[s] = fmaf(r01, vy, bx);
    oy[s] = fmaf(r11, vy, by);
    oz[s] = fmaf(r21, vy, bz);
  }
  if (g.flags & CJX_EWALD_SPHERE) {
    // the sphere's third coordinate w = lambda (u^2 + v^2) / (2 N pixel_size), rotated with R's third column
    const float cw = ewald_w(params + img, n);
    const float r02 = (float)R[2], r12 = (float)R[5], r22 = (float)R[8];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const float vy = (float)fft_index(act[s] ? vbase + 16 * s : 0, n);
      const float w = cw * fmaf(ux, ux, vy * vy);
      ox[s] = fmaf(r02, w, ox[s]);
      oy[s] = fmaf(r12, w, oy[s]);
      oz[s] = fmaf(r22, w, oz[s]);
    }
  }
  gather_samples<S>(grid, n, L, ox, oy, oz, act, wrap, g.fill, val);
  float2* col = hbuf + ((size_t)blockIdx.z * g.ncols + u) * g.ldh;
#pragma unroll
  for (int s = 0; s < S; ++s)
    if (act[s]) col[vbase + 16 * s] = val[s];
}

// The split gather for spline coefficients in the x-pair layout, four lanes
// per sample (sample_spline_team4), bound by the L1's data stage (80 % of its
// wavefronts, ncu, 64 images) next to the issue slots (65 %).  512 images 320^2 from
// N = 512: 3.13 ms with a lane per sample, 2.48 ms now; with 2, 3, 4 and 5
// CTAs per SM 3.30, 2.70, 2.48 and 2.98 ms (5 spill).  A warp takes 4 columns x 8 rows as four groups of 2 x 4 samples;
// the four lanes of a team then exchange their shares, so that lane t ends
// with the sample of group t, and store it.
// CTA patch: 16 columns x 16 steps rows: up to kSplineSteps steps, fewer where
// the tiles would not give every SM its 4 CTAs (spline_steps).  A warp of
// columns past the plane has nothing to do and returns.  With 4 steps always
// and those warps sampling: one image 320^2 from N = 512 22 us, 14 now (17 with
// a lane per sample), 2048 images 32^2 from N = 64 248 and 204 (360).
constexpr int kSplineSteps = 4;

static int spline_steps(dim3 tiles) {
  const int64_t all = (int64_t)tiles.x * tiles.y * tiles.z;
  return (int)std::max<int64_t>(1, std::min<int64_t>(kSplineSteps, all / (148 * 4)));
}

__global__ void __launch_bounds__(256, 4)
    k_gather_spline_team(const float4* __restrict__ coef, const cjx_image_params* __restrict__ params,
                         const int32_t* __restrict__ order, float2* __restrict__ hbuf, SliceGeom g, int64_t k0,
                         int steps) {
  const SplinePairLayout L(g.n);
  const int n = g.n;
  const int u0 = blockIdx.x * 16 + 4 * ((threadIdx.x >> 5) & 3);
  if (u0 >= g.ncols) return;  // the same for the whole warp; no barrier below
  const int64_t k = k0 + blockIdx.z;
  const int64_t img = order ? (int64_t)order[k] : k;
  const double* R = params[img].rot;
  const float r00 = (float)R[0], r01 = (float)R[1];
  const float r10 = (float)R[3], r11 = (float)R[4];
  const float r20 = (float)R[6], r21 = (float)R[7];
  const bool ewald = (g.flags & CJX_EWALD_SPHERE) != 0;
  float cw = 0.f, r02 = 0.f, r12 = 0.f, r22 = 0.f;
  if (ewald) {
    cw = ewald_w(params + img, n);
    r02 = (float)R[2];
    r12 = (float)R[5];
    r22 = (float)R[8];
  }
  const bool wrap = !(g.flags & CJX_ZERO_FILL_NEGATIVE);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = lane & 3, ly = t & 1, lz = t >> 1;
  const int su = (lane >> 2) & 1, sv = lane >> 3;
  float ux[2], bx[2], by[2], bz[2];  // the two columns this lane samples
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    ux[c] = (float)fft_index(min(u0 + 2 * c + su, g.ncols - 1), n);
    bx[c] = r00 * ux[c];
    by[c] = r10 * ux[c];
    bz[c] = r20 * ux[c];
  }
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    const int v0 = (blockIdx.y * steps + step) * 16 + 8 * (warp >> 2);
    if (v0 >= n) break;  // the same for the whole warp
    float2 p[4];
    // every lane samples (columns past the edge repeat the last, rows past N are low frequencies); only the stores
    // are guarded
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = q & 1;
      const float v = (float)(v0 + sv) + 4.0f * (q >> 1);
      const float vy = v < (float)(n - n / 2) ? v : v - (float)n;  // fft_index of the row
      float ox = fmaf(r01, vy, bx[c]), oy = fmaf(r11, vy, by[c]), oz = fmaf(r21, vy, bz[c]);
      if (ewald) {
        const float w = cw * fmaf(ux[c], ux[c], vy * vy);
        ox = fmaf(r02, w, ox);
        oy = fmaf(r12, w, oy);
        oz = fmaf(r22, w, oz);
      }
      p[q] = sample_spline_team4(coef, n, L, ox, oy, oz, wrap, g.fill, ly, lz);
    }
    float2 s[2];  // groups ly and ly + 2, summed over ly
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 give = ly ? p[2 * c] : p[2 * c + 1], own = ly ? p[2 * c + 1] : p[2 * c];
      s[c] = __fadd2_rn(own, make_float2(__shfl_xor_sync(0xffffffffu, give.x, 1),
                                         __shfl_xor_sync(0xffffffffu, give.y, 1)));
    }
    const float2 give = lz ? s[0] : s[1], own = lz ? s[1] : s[0];
    const float2 val = __fadd2_rn(own, make_float2(__shfl_xor_sync(0xffffffffu, give.x, 2),
                                                   __shfl_xor_sync(0xffffffffu, give.y, 2)));
    const int u = u0 + 2 * ly + su, v = v0 + 4 * lz + sv;
    if (u < g.ncols && v < n) hbuf[((size_t)blockIdx.z * g.ncols + u) * g.ldh + v] = val;
  }
}

template <bool PRIMES>
__global__ void __launch_bounds__(kWarps * 32, PRIMES ? 3 : 4)
    k_colifft_window(const float2* __restrict__ hbuf, float2* __restrict__ t1, const __grid_constant__ SliceGeom g) {
  extern __shared__ float2 smem[];
  const int n = g.n, h = n / 2;
  const int stride = 2 * n + 2;
  float2* tw = smem;
  float2* bufs = smem + n;
  build_twiddles(tw, n);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j0 = blockIdx.x * kWarps;
  const int j = j0 + warp;
  float2* a = bufs + warp * stride;
  float2* b = a + n;
  const bool ewald = (g.flags & CJX_EWALD_SPHERE) != 0;  // full complex surface: no Hermitian fix
  if (j < g.ncols) {
    const float2* col = hbuf + ((size_t)blockIdx.y * g.ncols + j) * g.ldh;
    for (int i = lane; i < n; i += 32) a[i] = col[i];
    __syncwarp();
    if (!ewald && (j == 0 || ((n % 2 == 0) && j == h))) {
      for (int i = lane; i <= n / 2; i += 32) {
        const int i2 = (i == 0) ? 0 : n - i;
        const float2 x = a[i], y = a[i2];
        const float2 sv = make_float2(0.5f * (x.x + y.x), 0.5f * (x.y - y.y));
        a[i] = sv;
        a[i2] = cconj(sv);
      }
      __syncwarp();
    }
    warp_fft<+1, PRIMES>(a, b, g.plan_n, tw, lane);
  }
  __syncthreads();
  const int res_off = (g.plan_n.nstages == 0 || (g.plan_n.nstages & 1)) ? n : 0;
  const int ncols = min(kWarps, g.ncols - j0);
  float2* dst = t1 + (size_t)blockIdx.y * g.py * g.ld1 + j0;
  for (int e = threadIdx.x; e < g.py * kWarps; e += blockDim.x) {
    const int m = e / kWarps, jj = e % kWarps;
    if (jj < ncols) {
      const int src = win_src(m, n, g.py, g.pad_left_y);
      dst[(size_t)m * g.ld1 + jj] = (src >= 0) ? bufs[jj * stride + res_off + src] : make_float2(0.f, 0.f);
    }
  }
}

// ---------------------------------------------------------------------------
// Pass B
// ---------------------------------------------------------------------------
template <bool PRIMES>
__global__ void __launch_bounds__(kWarps * 32, PRIMES ? 3 : 4)
    k_rows_c2r_r2c(const float2* __restrict__ t1, float2* __restrict__ t2, const __grid_constant__ SliceGeom g) {
  extern __shared__ float2 smem[];
  const int n = g.n, px = g.px;
  const int L = max(n, px);
  float2* twn = smem;
  float2* twp = twn + n;
  float2* bufs = twp + px;
  build_twiddles(twn, n);
  build_twiddles(twp, px);
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ra = 2 * (blockIdx.x * kWarps + warp);
  if (ra >= g.py) return;
  const bool has_b = (ra + 1) < g.py;
  float2* a = bufs + warp * (2 * L + 2);
  float2* b = a + L;
  const float2* rowA = t1 + ((size_t)blockIdx.y * g.py + ra) * g.ld1;
  const float2* rowB = rowA + g.ld1;

  // Z = A + iB on the Hermitian extension; DC and (even N) Nyquist bins use
  // the real part only, as an irfft does.
  const int h = n / 2;
  for (int k = lane; k <= h; k += 32) {
    float2 A = rowA[k];
    float2 B = has_b ? rowB[k] : make_float2(0.f, 0.f);
    if (k == 0 || ((n % 2 == 0) && k == h)) {
      a[k] = make_float2(A.x, B.x);
    } else {
      a[k] = make_float2(A.x - B.y, A.y + B.x);
      a[n - k] = make_float2(A.x + B.y, B.x - A.y);
    }
  }
  __syncwarp();
  float2* z = warp_fft<+1, PRIMES>(a, b, g.plan_n, twn, lane);  // z = a_row + i b_row (real rows)
  float2* w = (z == a) ? b : a;
  for (int m = lane; m < px; m += 32) {
    const int src = win_src(m, n, px, g.pad_left_x);
    w[m] = (src >= 0) ? z[src] : make_float2(0.f, 0.f);
  }
  __syncwarp();
  float2* W = warp_fft<-1, PRIMES>(w, z, g.plan_px, twp, lane);
  float2* outA = t2 + ((size_t)blockIdx.y * g.py + ra) * g.ld2;
  for (int k = lane; k < g.pxh; k += 32) {
    const float2 Wk = W[k];
    const float2 Wm = W[k == 0 ? 0 : px - k];
    outA[k] = make_float2(0.5f * (Wk.x + Wm.x), 0.5f * (Wk.y - Wm.y));
    if (has_b) outA[g.ld2 + k] = make_float2(0.5f * (Wk.y + Wm.y), -0.5f * (Wk.x - Wm.x));
  }
}

// ---------------------------------------------------------------------------
// Pass C
// ---------------------------------------------------------------------------
template <bool PRIMES>
__global__ void __launch_bounds__(kWarps * 32, PRIMES ? 3 : 4)
    k_colfft_epilogue(const float2* __restrict__ t2, const cjx_image_params* __restrict__ params,
                      const int32_t* __restrict__ order, float2* __restrict__ out, const __grid_constant__ SliceGeom g, int64_t k0,
                      float norm) {
  extern __shared__ float2 smem[];
  const int py = g.py;
  const int stride = 2 * py + 2;
  float2* tw = smem;
  float2* bufs = smem + py;
  ImageConsts& sc = *reinterpret_cast<ImageConsts*>(bufs + kWarps * stride);
  build_twiddles(tw, py);

  const int j0 = blockIdx.x * kWarps;
  const int ncols = min(kWarps, g.pxh - j0);
  const float2* src = t2 + (size_t)blockIdx.y * py * g.ld2 + j0;
  for (int e = threadIdx.x; e < py * kWarps; e += blockDim.x) {
    const int m = e / kWarps, jj = e % kWarps;
    if (jj < ncols) bufs[jj * stride + m] = src[(size_t)m * g.ld2 + jj];
  }
  const int64_t k = k0 + blockIdx.y;
  const int64_t img = order ? (int64_t)order[k] : k;
  // once per CTA: its double divisions and sincos in every thread took as long as the transforms
  if (threadIdx.x == 0) sc = load_image_consts(params + img, norm, g.py, g.px);
  __syncthreads();
  const ImageConsts& c = sc;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < ncols) {
    float2* a = bufs + warp * stride;
    float2* X = warp_fft<-1, PRIMES>(a, a + py, g.plan_py, tw, lane);
    const int j = j0 + warp;
    for (int i = lane; i < py; i += 32) X[i] = apply_filter(apply_epilogue(X[i], i, j, py, g.px, g.flags, c), g, i, j, g.pxh);
  }
  __syncthreads();
  const int res_off = (g.plan_py.nstages == 0 || (g.plan_py.nstages & 1)) ? py : 0;
  float2* dst = out + (size_t)img * py * g.pxh + j0;
  for (int e = threadIdx.x; e < py * kWarps; e += blockDim.x) {
    const int m = e / kWarps, jj = e % kWarps;
    if (jj < ncols) dst[(size_t)m * g.pxh + jj] = bufs[jj * stride + res_off + m];
  }
}

// ---------------------------------------------------------------------------
// Register-FFT forms of the three resize passes (n = 32 R sizes).  Same data
// flow as the shared-memory Stockham kernels above; the transforms run in
// registers with warp shuffles (cjx_fft.cuh) and shared memory only holds
// twiddle tables and the transposes (padded layout pad16).
// ---------------------------------------------------------------------------

// Pass A (split): column inverse FFT + window of the gathered slice H.
template <int R, bool T512 = false>
__global__ void __launch_bounds__(kWarps * 32)
    k_colifft_window_reg(const float2* __restrict__ hbuf, float2* __restrict__ t1, SliceGeom g) {
  constexpr int n = 32 * R;
  constexpr int stride = pad16(n) + 1;
  extern __shared__ float2 smem[];
  __shared__ float2 w32[32];
  float2* tab = smem;
  float2* bufs = smem + n;
  int* winy = reinterpret_cast<int*>(bufs + kWarps * stride);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j0 = blockIdx.x * kWarps;
  const int j = j0 + warp;
  float2* buf = bufs + warp * stride;
  const int bl = T512 ? lane : brev5(lane);  // the transpose FFT takes natural lane order
  float2 x[R];
  // table copy first: here (one column per warp, loaded straight into
  // registers) that measured 1.3 % faster than issuing the column loads first
  build_reg_twiddles(tab, n);
  build_w32(w32);
  if (j < g.ncols) {
    const float2* col = hbuf + ((size_t)blockIdx.y * g.ncols + j) * g.ldh;
    // the Ewald sphere's full complex surface takes no Hermitian fix
    const bool sym = !(g.flags & CJX_EWALD_SPHERE) && ((j == 0) || (j == n / 2));
#pragma unroll
    for (int n1 = 0; n1 < R; ++n1) {
      const int idx = 32 * n1 + bl;
      float2 v = col[idx];
      if (sym) {  // (S[v] + conj(S[-v])) / 2, as the irfftn of the reference sees it
        const float2 m = col[idx == 0 ? 0 : n - idx];
        v = make_float2(0.5f * (v.x + m.x), 0.5f * (v.y - m.y));
      }
      x[n1] = v;
    }
  }
  __syncthreads();
  if (j < g.ncols) {
    const LaneTwiddles lt = make_lane_twiddles(w32, lane);
    if constexpr (T512) {
      static_assert(R == 16, "the transpose FFT is 512-point");
      warp_fft512_t<+1>(x, tab, w32, buf, lane);
#pragma unroll
      for (int q = 0; q < R; ++q) buf[pad16(fft512_t_out(q, lane))] = x[q];
    } else {
      warp_fft_reg<R, +1>(x, tab, lt, lane);
#pragma unroll
      for (int k1 = 0; k1 < R; ++k1) buf[pad16(k1 + R * lane)] = x[k1];
    }
  }
  // the window's map last: its place among the loads decided the pass's time (1024 images 320^2 from N = 512: 490
  // us there with divisions in win_src, 508 without, 492 here; 8192 images 64^2 from N = 128 286, 278, 273)
  for (int m = threadIdx.x; m < g.py; m += blockDim.x) winy[m] = win_src(m, n, g.py, g.pad_left_y);
  __syncthreads();
  const int ncols = min(kWarps, g.ncols - j0);
  float2* dst = t1 + (size_t)blockIdx.y * g.py * g.ld1 + j0;
  for (int e = threadIdx.x; e < g.py * kWarps; e += blockDim.x) {
    const int m = e / kWarps, jj = e % kWarps;
    if (jj < ncols) {
      const int src = winy[m];
      dst[(size_t)m * g.ld1 + jj] = (src >= 0) ? bufs[jj * stride + pad16(src)] : make_float2(0.f, 0.f);
    }
  }
}

// Pass B: two rows per warp.  N-point inverse FFT of A + iB (register form,
// R = RN), Px window, Px-point forward FFT (register form, RP), split.
// The load of the packed pair (z = A + iB in the lane's bit-reversed order)
// is separate, so that a kernel can issue it before its table copy.
// Per-warp buffer of the row pass: the N-point transform's staging (stage512
// with the transpose FFT, pad16 otherwise) and the Px-point one's (stage_r).
__host__ __device__ inline int rows_stride(int n, int px, bool t512) {
  const int sn = t512 ? kStage512Size : pad16(n - 1) + 1;
  const int sp = stage_r_size(px / 32);
  return (sn > sp ? sn : sp) + 1;
}

template <int RN, bool NATURAL = false>
__device__ __forceinline__ void rows_pair_load(const float2* __restrict__ rowA, const float2* __restrict__ rowB,
                                               bool has_b, float2 (&z)[RN], int lane) {
  constexpr int n = 32 * RN, h = n / 2;
  const int bl = NATURAL ? lane : brev5(lane);  // natural lane order feeds the transpose FFT
#pragma unroll
  for (int n1 = 0; n1 < RN; ++n1) {
    const int idx = 32 * n1 + bl;
    if (idx == 0 || idx == h) {
      const float2 A = rowA[idx];
      const float2 B = has_b ? rowB[idx] : make_float2(0.f, 0.f);
      z[n1] = make_float2(A.x, B.x);
    } else if (idx < h) {
      const float2 A = rowA[idx];
      const float2 B = has_b ? rowB[idx] : make_float2(0.f, 0.f);
      z[n1] = make_float2(A.x - B.y, A.y + B.x);
    } else {
      const float2 A = rowA[n - idx];
      const float2 B = has_b ? rowB[n - idx] : make_float2(0.f, 0.f);
      z[n1] = make_float2(A.x + B.y, B.x - A.y);
    }
  }
}

template <int RN, int RP, bool T512 = false>
__device__ __forceinline__ void rows_pair_reg(float2 (&z)[RN], bool has_b, float2* __restrict__ outA, int ld2,
                                              float2* buf, const float2* tabN, const float2* tabP,
                                              const LaneTwiddles& lt, int lane, const int* winx,
                                              const float2* w32 = nullptr) {
  constexpr int px = 32 * RP;
  const int bl = brev5(lane);
  if constexpr (T512) {  // 512-point inverse as 16 x 32 through one shared-memory transpose (z in natural order)
    static_assert(RN == 16, "the transpose FFT is 512-point");
    warp_fft512_t<+1>(z, tabN, w32, buf, lane);
#pragma unroll
    for (int q = 0; q < RN; ++q) buf[stage512(fft512_t_out(q, lane))] = z[q];
  } else {
    warp_fft_reg<RN, +1>(z, tabN, lt, lane);  // z = a + i b (the two real rows)
#pragma unroll
    for (int k1 = 0; k1 < RN; ++k1) buf[pad16(k1 + RN * lane)] = z[k1];
  }
  __syncwarp();
  float2 w[RP];
#pragma unroll
  for (int n1 = 0; n1 < RP; ++n1) {
    const int src = winx[32 * n1 + bl];
    w[n1] = (src >= 0) ? buf[T512 ? stage512(src) : pad16(src)] : make_float2(0.f, 0.f);
  }
  __syncwarp();
  warp_fft_reg<RP, -1>(w, tabP, lt, lane);
#pragma unroll
  for (int k1 = 0; k1 < RP; ++k1) buf[stage_r(RP, k1 + RP * lane)] = w[k1];
  __syncwarp();
  for (int k = lane; k <= px / 2; k += 32) {
    const float2 Wk = buf[stage_r(RP, k)];
    const float2 Wm = buf[stage_r(RP, k == 0 ? 0 : px - k)];
    outA[k] = make_float2(0.5f * (Wk.x + Wm.x), 0.5f * (Wk.y - Wm.y));
    if (has_b) outA[ld2 + k] = make_float2(0.5f * (Wk.y + Wm.y), -0.5f * (Wk.x - Wm.x));
  }
}

// Body of the row pass for the CTA at (bx, by) of its launch: smem is the
// dynamic shared memory, w32 a 32-entry shared table.
template <int RN, bool T512>
__device__ __forceinline__ void rows_reg_body(const float2* __restrict__ t1, float2* __restrict__ t2,
                                              const SliceGeom& g, int rp, int bx, int by, float2* smem, float2* w32) {
  constexpr int n = 32 * RN;
  const int px = g.px;
  const int stride = rows_stride(n, px, T512);
  float2* tabN = smem;
  float2* tabP = tabN + n;
  float2* bufs = tabP + px;
  int* winx = reinterpret_cast<int*>(bufs + kWarps * stride);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ra = 2 * (bx * kWarps + warp);
  const bool has_b = (ra + 1) < g.py;
  // the row pair is loaded first, so that its latency overlaps the table copy
  float2 z[RN];
  if (ra < g.py) {
    const float2* rowA = t1 + ((size_t)by * g.py + ra) * g.ld1;
    rows_pair_load<RN, T512>(rowA, rowA + g.ld1, has_b, z, lane);
  }
  build_reg_twiddles(tabN, n);
  build_reg_twiddles(tabP, px);
  build_w32(w32);
  for (int m = threadIdx.x; m < px; m += blockDim.x) winx[m] = win_src(m, n, px, g.pad_left_x);
  __syncthreads();
  if (ra >= g.py) return;
  float2* outA = t2 + ((size_t)by * g.py + ra) * g.ld2;
  float2* buf = bufs + warp * stride;
  const LaneTwiddles lt = make_lane_twiddles(w32, lane);
  switch (rp) {
#define CJX_ROWS_CASE(RPV) \
  case RPV: rows_pair_reg<RN, RPV, T512>(z, has_b, outA, g.ld2, buf, tabN, tabP, lt, lane, winx, w32); break;
    CJX_ROWS_CASE(1) CJX_ROWS_CASE(2) CJX_ROWS_CASE(3) CJX_ROWS_CASE(4) CJX_ROWS_CASE(5)
    CJX_ROWS_CASE(6) CJX_ROWS_CASE(8) CJX_ROWS_CASE(10) CJX_ROWS_CASE(12) CJX_ROWS_CASE(16)
#undef CJX_ROWS_CASE
    default: break;
  }
}

template <int RN, bool T512 = false>
__global__ void __launch_bounds__(kWarps * 32, 4)
    k_rows_reg(const float2* __restrict__ t1, float2* __restrict__ t2, SliceGeom g, int rp) {
  extern __shared__ float2 smem[];
  __shared__ float2 w32[32];
  rows_reg_body<RN, T512>(t1, t2, g, rp, blockIdx.x, blockIdx.y, smem, w32);
}

// Pass C: column forward FFT of T2 + epilogue.  Body for the CTA at (bx, by):
// smem is the dynamic shared memory, w32 and sc shared scratch.
template <int R>
__device__ __forceinline__ void colfft_epilogue_body(const float2* __restrict__ t2,
                                                     const cjx_image_params* __restrict__ params,
                                                     const int32_t* __restrict__ order, float2* __restrict__ out,
                                                     const SliceGeom& g, int64_t k0, float norm, int bx, int by,
                                                     float2* smem, float2* w32, ImageConsts& sc) {
  constexpr int py = 32 * R;
  constexpr int stride = stage_r_size(R) + 1;
  float2* tab = smem;
  float2* row_phase = smem + py;  // exp(-2 pi i qy(i) ty)
  float2* bufs = smem + 2 * py;
  const int j0 = bx * kWarps;
  const int ncols = min(kWarps, g.pxh - j0);
  const float2* src = t2 + (size_t)by * py * g.ld2 + j0;
  // staging: thread t moves column t % kWarps, rows t / kWarps + 32 q; all R
  // loads are issued before the table copy and the shared-memory stores
  static_assert(kWarps * 32 == 256, "the staging map assumes 256 threads");
  const int sj = threadIdx.x % kWarps, sm0 = threadIdx.x / kWarps;
  float2 st[R];
  if (sj < ncols) {
#pragma unroll
    for (int q = 0; q < R; ++q) st[q] = src[(size_t)(sm0 + 32 * q) * g.ld2 + sj];
  }
  build_reg_twiddles(tab, py);
  build_w32(w32);
  if (sj < ncols) {
#pragma unroll
    for (int q = 0; q < R; ++q) bufs[sj * stride + pad16(sm0 + 32 * q)] = st[q];
  }
  const int64_t k = k0 + by;
  const int64_t img = order ? (int64_t)order[k] : k;
  // the image's constants (double divisions and a sincos) once per CTA, not once per thread
  if (threadIdx.x == 0) sc = load_image_consts(params + img, norm, g.py, g.px);
  __syncthreads();
  const ImageConsts& c = sc;  // read from shared memory where used (keeps the register count down)
  if (g.flags & CJX_APPLY_TRANSLATION)
    for (int i = threadIdx.x; i < py; i += blockDim.x) row_phase[i] = phase_factor((double)fft_index(i, py) * c.qy_step * c.ty);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < ncols) {
    float2* buf = bufs + warp * stride;
    const LaneTwiddles lt = make_lane_twiddles(w32, lane);
    const int bl = brev5(lane);
    float2 x[R];
#pragma unroll
    for (int n1 = 0; n1 < R; ++n1) x[n1] = buf[pad16(32 * n1 + bl)];
    warp_fft_reg<R, -1>(x, tab, lt, lane);
    const int j = j0 + warp;
    const ColumnEpilogue ce = column_epilogue(j, g.flags, c);
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < R; ++k1) {
      const int i = k1 + R * lane;
      buf[stage_r(R, i)] =
          apply_filter(apply_column_epilogue(x[k1], i, j, py, g.px, g.flags, c, ce, row_phase), g, i, j, g.pxh);
    }
  }
  __syncthreads();
  float2* dst = out + (size_t)img * py * g.pxh + j0;
  for (int e = threadIdx.x; e < py * kWarps; e += blockDim.x) {
    const int m = e / kWarps, jj = e % kWarps;
    if (jj < ncols) dst[(size_t)m * g.pxh + jj] = bufs[jj * stride + stage_r(R, m)];
  }
}

template <int R>
__global__ void __launch_bounds__(kWarps * 32)
    k_colfft_epilogue_reg(const float2* __restrict__ t2, const cjx_image_params* __restrict__ params,
                          const int32_t* __restrict__ order, float2* __restrict__ out, SliceGeom g, int64_t k0,
                          float norm) {
  extern __shared__ float2 smem[];
  __shared__ float2 w32[32];
  __shared__ ImageConsts sc;
  colfft_epilogue_body<R>(t2, params, order, out, g, k0, norm, blockIdx.x, blockIdx.y, smem, w32, sc);
}

// ---------------------------------------------------------------------------
// Row and column passes for every group of a wave in one launch each.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kWarps * 32, 3) k_rows_wave(const __grid_constant__ Wave w) {
  extern __shared__ float2 smem[];
  __shared__ float2 w32[32];
  const int gi = wave_group(w, 1, blockIdx.x);
  const WaveGroup& q = w.grp[gi];
  const int local = blockIdx.x - q.cta0[1];
  const int cx = (q.g.py + 2 * kWarps - 1) / (2 * kWarps);
  const int bx = local % cx, by = local / cx;
  const int rp = reg_fft_radix(q.g.px);
  switch (reg_fft_radix(q.g.n)) {
#define CJX_RW(R) \
  case R: rows_reg_body<R, false>(q.t1, q.t2, q.g, rp, bx, by, smem, w32); break;
    CJX_RW(1) CJX_RW(2) CJX_RW(3) CJX_RW(4) CJX_RW(5) CJX_RW(6) CJX_RW(8) CJX_RW(10) CJX_RW(12)
#undef CJX_RW
    case 16:
      if (w.rows_t512)
        rows_reg_body<16, true>(q.t1, q.t2, q.g, rp, bx, by, smem, w32);
      else
        rows_reg_body<16, false>(q.t1, q.t2, q.g, rp, bx, by, smem, w32);
      break;
    default:
      break;
  }
}

__global__ void __launch_bounds__(kWarps * 32, 3) k_tail_wave(const __grid_constant__ Wave w) {
  extern __shared__ float2 smem[];
  __shared__ float2 w32[32];
  __shared__ ImageConsts sc;
  const int gi = wave_group(w, 2, blockIdx.x);
  const WaveGroup& q = w.grp[gi];
  const int local = blockIdx.x - q.cta0[2];
  const int cx = (q.g.pxh + kWarps - 1) / kWarps;
  const int bx = local % cx, by = local / cx;
  const float norm = (float)(1.0 / ((double)q.g.n * (double)q.g.n));
  switch (reg_fft_radix(q.g.py)) {
#define CJX_TW(R) \
  case R: colfft_epilogue_body<R>(q.t2, q.params, q.order, q.out, q.g, q.k0, norm, bx, by, smem, w32, sc); break;
    CJX_TW(1) CJX_TW(2) CJX_TW(3) CJX_TW(4) CJX_TW(5) CJX_TW(6) CJX_TW(8) CJX_TW(10) CJX_TW(12) CJX_TW(16)
#undef CJX_TW
    default:
      break;
  }
}

// ---------------------------------------------------------------------------
// No-resize path: fused slice + epilogue, one thread per output pixel.
// ---------------------------------------------------------------------------
template <typename Layout>
__global__ void __launch_bounds__(256)
    k_slice_direct(const float2* __restrict__ grid, const cjx_image_params* __restrict__ params,
                   const int32_t* __restrict__ order, float2* __restrict__ out, SliceGeom g, int64_t k0) {
  const Layout L(g.n);
  const int n = g.n, h = n / 2;
  const int64_t k = k0 + blockIdx.y;
  const int64_t img = order ? (int64_t)order[k] : k;
  const double* R = params[img].rot;
  const float r00 = (float)R[0], r01 = (float)R[1];
  const float r10 = (float)R[3], r11 = (float)R[4];
  const float r20 = (float)R[6], r21 = (float)R[7];
  const bool wrap = !(g.flags & CJX_ZERO_FILL_NEGATIVE);
  const ImageConsts c = load_image_consts(params + img, 1.0f, n, n);
  const int total = n * g.nxh;
  float2* dst = out + (size_t)img * total;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int i = e / g.nxh, j = e - i * g.nxh;
    const float ux = (float)fft_index(j, n), vy = (float)fft_index(i, n);
    const float ox = fmaf(r01, vy, r00 * ux), oy = fmaf(r11, vy, r10 * ux), oz = fmaf(r21, vy, r20 * ux);
    const bool act = true;
    float2 v;
    gather_samples<1>(grid, n, L, &ox, &oy, &oz, &act, wrap, g.fill, &v);
    // convert_fftn_to_rfftn(mode="real")  (cryojax/ndimage/_fourier_utils.py:6-57)
    if ((n % 2 == 0) && ((i == h && j == 0) || (i == 0 && j == h) || (i == h && j == h))) v.y = 0.f;
    dst[e] = apply_filter(apply_epilogue(v, i, j, n, n, g.flags, c), g, i, j, g.nxh);
  }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
static size_t smem_a(const SliceGeom& g) { return sizeof(float2) * (size_t)(g.n + kWarps * (2 * g.n + 2)); }
static size_t smem_b(const SliceGeom& g) {
  const int L = std::max(g.n, g.px);
  return sizeof(float2) * (size_t)(g.n + g.px + kWarps * (2 * L + 2));
}
static size_t smem_c(const SliceGeom& g) {
  return sizeof(float2) * (size_t)(g.py + kWarps * (2 * g.py + 2)) + sizeof(ImageConsts);
}

// Process-wide tuning knobs (cjx_tuning_set / cjx_tuning_get).
static std::atomic<int64_t> g_gather_ilp{2};
static std::atomic<int64_t> g_chunk_bytes{2048ll << 20};  // 16384 images 320^2 from N = 512: 36.2 ms per step, 36.9 at 1 GiB
static std::atomic<int64_t> g_gather_mode{2};  // 16384 images 320^2 from N = 512: 37.0 ms per step against 42.2 split
static std::atomic<int64_t> g_fft_mode{3};  // 16384 images 320^2 from N = 512: row pass 7.5 ms against 7.9
static std::atomic<int64_t> g_gather_tile{1};
static std::atomic<int64_t> g_scatter_vec{1};
static std::atomic<int64_t> g_spline_ilp{4};
static std::atomic<int64_t> g_multi_waves{0};

static int round_up(int x, int m) { return (x + m - 1) / m * m; }

int make_geom(const cjx_slice_desc* d, SliceGeom* g) {
  if (!d) return fail(CJX_ERR_INVALID_ARGUMENT, "desc is NULL");
  if (d->n < 2 || d->py < 1 || d->px < 2)
    return fail(CJX_ERR_INVALID_ARGUMENT, "need n >= 2, py >= 1, px >= 2");
  if (d->n > CJX_MAX_SIDE || d->py > CJX_MAX_SIDE || d->px > CJX_MAX_SIDE)
    return fail(CJX_ERR_UNSUPPORTED, "volume side and image sides are limited to CJX_MAX_SIDE");
  const uint32_t known =
      CJX_APPLY_CTF | CJX_APPLY_TRANSLATION | CJX_APPLY_ENVELOPE | CJX_ZERO_FILL_NEGATIVE | CJX_GRID_BRICKED |
      CJX_GRID_BRICKED_PAIRS | CJX_GRID_SPLINE | CJX_EWALD_SPHERE;
  if (d->flags & ~known) return fail(CJX_ERR_INVALID_ARGUMENT, "unknown flag bits");
  if ((d->flags & CJX_EWALD_SPHERE) && !(d->flags & CJX_APPLY_CTF) &&
      (d->flags & (CJX_APPLY_ENVELOPE | CJX_APPLY_TRANSLATION)))
    return fail(CJX_ERR_INVALID_ARGUMENT,
                "CJX_EWALD_SPHERE without CJX_APPLY_CTF outputs the full spectrum: no envelope or translation");
  if ((d->flags & CJX_GRID_BRICKED) && (d->flags & CJX_GRID_BRICKED_PAIRS))
    return fail(CJX_ERR_INVALID_ARGUMENT, "CJX_GRID_BRICKED and CJX_GRID_BRICKED_PAIRS are exclusive");
  g->n = d->n;
  g->py = d->py;
  g->px = d->px;
  g->nxh = d->n / 2 + 1;
  g->pxh = d->px / 2 + 1;
  const bool ewald = (d->flags & CJX_EWALD_SPHERE) != 0;
  g->ncols = ewald ? d->n : g->nxh;
  g->ld1 = round_up(g->ncols, 8);
  g->ld2 = round_up(ewald ? d->px : g->pxh, 8);
  g->ldh = round_up(g->n, 8);
  auto left_pad = [](int pad_dim, int image_dim) {
    const int pad = pad_dim - image_dim;
    if (pad_dim % 2 == 0 && image_dim % 2 == 1) return pad / 2 + 1;
    return pad / 2;
  };
  g->pad_left_y = d->py > d->n ? left_pad(d->py, d->n) : 0;
  g->pad_left_x = d->px > d->n ? left_pad(d->px, d->n) : 0;
  g->flags = d->flags;
  g->fill = make_float2(d->fill_re, d->fill_im);
  g->filter = nullptr;
  g->plan_n = make_fft_plan(d->n);
  g->plan_py = make_fft_plan(d->py);
  g->plan_px = make_fft_plan(d->px);
  return CJX_OK;
}

bool needs_resize(const SliceGeom& g) { return !(g.py == g.n && g.px == g.n); }

// Per image: T1 [Py][ld1], T2 [Py][ld2] and the split gather's H [ncols][ldh].
size_t workspace_per_image(const SliceGeom& g) {
  return sizeof(float2) * ((size_t)g.py * g.ld1 + (size_t)g.py * g.ld2 + (size_t)g.ncols * g.ldh);
}

// Default chunk: CJX_TUNE_CHUNK_BYTES of intermediates (1 GiB unless set); larger
// chunks mean fewer launches and shorter tails, at the cost of workspace.
int64_t default_chunk(const SliceGeom& g, int64_t n_images) {
  const size_t per = workspace_per_image(g);
  int64_t c = (int64_t)((size_t)g_chunk_bytes.load() / std::max<size_t>(per, 1));
  c = std::max<int64_t>(c, 1);
  c = std::min<int64_t>(c, 65535);
  return std::min<int64_t>(c, std::max<int64_t>(n_images, 1));
}

// Process-wide tuning knobs (cjx_tuning_set / cjx_tuning_get), declared above.

int64_t tuning_get(int key) {
  if (key == CJX_TUNE_GATHER_ILP) return g_gather_ilp.load();
  if (key == CJX_TUNE_CHUNK_BYTES) return g_chunk_bytes.load();
  if (key == CJX_TUNE_GATHER_MODE) return g_gather_mode.load();
  if (key == CJX_TUNE_FFT_MODE) return g_fft_mode.load();
  if (key == CJX_TUNE_GATHER_TILE) return g_gather_tile.load();
  if (key == CJX_TUNE_SCATTER_VEC) return g_scatter_vec.load();
  if (key == CJX_TUNE_SPLINE_ILP) return g_spline_ilp.load();
  if (key == CJX_TUNE_MULTI_WAVES) return g_multi_waves.load();
  return -1;
}

int tuning_set(int key, int64_t value) {
  if (key == CJX_TUNE_GATHER_ILP) {
    if (value != 1 && value != 2 && value != 4) return fail(CJX_ERR_INVALID_ARGUMENT, "gather ILP must be 1, 2 or 4");
    g_gather_ilp = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_CHUNK_BYTES) {
    if (value < (1 << 20)) return fail(CJX_ERR_INVALID_ARGUMENT, "chunk bytes must be >= 1 MiB");
    g_chunk_bytes = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_GATHER_MODE) {
    if (value < 0 || value > 2) return fail(CJX_ERR_INVALID_ARGUMENT, "gather mode must be 0, 1 or 2");
    g_gather_mode = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_FFT_MODE) {
    if (value < 0 || value > 3) return fail(CJX_ERR_INVALID_ARGUMENT, "FFT mode must be 0, 1, 2 or 3");
    g_fft_mode = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_GATHER_TILE) {
    if (value < 0 || value > 3) return fail(CJX_ERR_INVALID_ARGUMENT, "gather tile must be 0, 1, 2 or 3");
    g_gather_tile = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_SPLINE_ILP) {
    if (value != 1 && value != 2 && value != 4) return fail(CJX_ERR_INVALID_ARGUMENT, "spline ILP must be 1, 2 or 4");
    g_spline_ilp = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_MULTI_WAVES) {
    if (value != 0 && value != 1) return fail(CJX_ERR_INVALID_ARGUMENT, "multi waves must be 0 or 1");
    g_multi_waves = value;
    return CJX_OK;
  }
  if (key == CJX_TUNE_SCATTER_VEC) {
    if (value < 0 || value > 2) return fail(CJX_ERR_INVALID_ARGUMENT, "scatter mode must be 0, 1 or 2");
    g_scatter_vec = value;
    return CJX_OK;
  }
  return fail(CJX_ERR_INVALID_ARGUMENT, "unknown tuning key");
}

template <typename K>
static cudaError_t allow_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

static int ensure_smem_attrs() {
  static PerDeviceOnce once;
  const cudaError_t e = once.run([] {
    cudaError_t e = cudaSuccess;
#define CJX_SMEM_ATTR(P)                                                             \
  if (e == cudaSuccess) e = allow_smem(k_gather_colifft<1, LinearLayout, P>);        \
  if (e == cudaSuccess) e = allow_smem(k_gather_colifft<2, LinearLayout, P>);        \
  if (e == cudaSuccess) e = allow_smem(k_gather_colifft<4, LinearLayout, P>);        \
  if (e == cudaSuccess) e = allow_smem(k_gather_colifft<1, BrickLayout, P>);         \
  if (e == cudaSuccess) e = allow_smem(k_gather_colifft<2, BrickLayout, P>);         \
  if (e == cudaSuccess) e = allow_smem(k_gather_colifft<4, BrickLayout, P>);         \
  if (e == cudaSuccess) e = allow_smem(k_colifft_window<P>);                         \
  if (e == cudaSuccess) e = allow_smem(k_rows_c2r_r2c<P>);                           \
  if (e == cudaSuccess) e = allow_smem(k_colfft_epilogue<P>);
    CJX_SMEM_ATTR(false) CJX_SMEM_ATTR(true)
#undef CJX_SMEM_ATTR
    return e;
  });
  return e == cudaSuccess ? CJX_OK : check_cuda(e, "cudaFuncSetAttribute (slice kernels)");
}

int launch_ewald_rows(const SliceGeom& g, const float2* t1, float2* t2, int cnt, cudaStream_t stream,
                      const Tuning& tn);
bool fused_gather_supported(const SliceGeom& g);
int launch_gather_colifft_fused(const SliceGeom& g, const float2* grid, const cjx_image_params* params,
                                const int32_t* order, int64_t k0, int cnt, float2* t1, const Tuning& tn,
                                cudaStream_t stream);
int launch_ewald_colfft(const SliceGeom& g, const float2* t2, const cjx_image_params* params, const int32_t* order,
                        float2* out, int64_t k0, int cnt, cudaStream_t stream, const Tuning& tn);
int launch_ewald_direct(const SliceGeom& g, const float2* grid, const cjx_image_params* params, const int32_t* order,
                        int64_t n_images, float2* out, cudaStream_t stream);

// The front of the resize path for one chunk of `cnt` images starting at
// processing index k0: gather and column inverse FFT + window, into T1.
static int launch_front(const SliceGeom& g, const float2* grid, const cjx_image_params* params, const int32_t* order,
                        int64_t k0, int cnt, float2* t1, float2* hb, cudaStream_t stream, const Tuning& tn) {
  if (int e = ensure_smem_attrs()) return e;
  const int64_t ilp = (g.flags & CJX_GRID_SPLINE) ? tn.spline_ilp : tn.ilp;
  const int rn = reg_fft_radix(g.n);
  const bool fast = tn.fft_mode >= 1;
  // gather mode 2: the register-FFT fused pass (trilinear grids, N = 32 R); otherwise the split pair of
  // kernels, or mode 0's shared-memory fused kernel, which has no pair, spline or Ewald path
  const bool fused_reg = tn.gather_mode == 2 && fast && fused_gather_supported(g);
  const bool split = !fused_reg && (tn.gather_mode != 0 ||
                                    (g.flags & (CJX_GRID_BRICKED_PAIRS | CJX_GRID_SPLINE | CJX_EWALD_SPHERE)));
  const bool t512 = tn.fft_mode >= 2 && rn == 16;  // 512-point column transforms through the transpose FFT
  const size_t sa = smem_a(g);
  const size_t sa_reg = sizeof(float2) * (size_t)(g.n + kWarps * (pad16(g.n) + 1)) + sizeof(int) * (size_t)g.py;
    if (fused_reg) {
      if (int e = launch_gather_colifft_fused(g, grid, params, order, k0, cnt, t1, tn, stream)) return e;
    } else if (split) {
      const dim3 gg((g.ncols + 15) / 16, (g.n + 16 * (int)ilp - 1) / (16 * (int)ilp), cnt);
      prof_begin(stream);
      const bool bricked = (g.flags & CJX_GRID_BRICKED) != 0;
      const bool pairs = (g.flags & CJX_GRID_BRICKED_PAIRS) != 0;
      const bool spline = (g.flags & CJX_GRID_SPLINE) != 0;
      const int64_t map = tn.tile;
#define CJX_GSM(S, M)                                                                                   \
  if (spline && bricked)                                                                           \
    k_gather_slice<S, SplineBrickLayout, M><<<gg, 256, 0, stream>>>(grid, params, order, hb, g, k0);  \
  else if (spline)                                                                                      \
    k_gather_slice<S, SplineLinearLayout, M><<<gg, 256, 0, stream>>>(grid, params, order, hb, g, k0); \
  else if (pairs)                                                                                   \
    k_gather_slice<S, PairLayout, M><<<gg, 256, 0, stream>>>(grid, params, order, hb, g, k0);   \
  else if (bricked)                                                                                 \
    k_gather_slice<S, BrickLayout, M><<<gg, 256, 0, stream>>>(grid, params, order, hb, g, k0);  \
  else                                                                                              \
    k_gather_slice<S, LinearLayout, M><<<gg, 256, 0, stream>>>(grid, params, order, hb, g, k0);
#define CJX_GS(S)       \
  if (map == 1) {       \
    CJX_GSM(S, 1)       \
  } else if (map == 2) { \
    CJX_GSM(S, 2)       \
  } else {              \
    CJX_GSM(S, 0)       \
  }
      if (spline && pairs) {
        dim3 gt((g.ncols + 15) / 16, (g.n + 15) / 16, cnt);
        const int steps = spline_steps(gt);
        gt.y = (gt.y + steps - 1) / steps;
        k_gather_spline_team<<<gt, 256, 0, stream>>>(reinterpret_cast<const float4*>(grid), params, order, hb, g, k0,
                                                     steps);
      } else if (ilp == 4) {
        CJX_GS(4)
      } else if (ilp == 2) {
        CJX_GS(2)
      } else {
        CJX_GS(1)
      }
#undef CJX_GS
#undef CJX_GSM
      prof_end(spline && pairs ? "k_gather_spline_team" : "k_gather_slice", stream);
      prof_begin(stream);
      const dim3 gc((g.ncols + kWarps - 1) / kWarps, cnt);
      if (fast && t512) {
        k_colifft_window_reg<16, true><<<gc, kWarps * 32, sa_reg, stream>>>(hb, t1, g);
      } else if (fast && rn) {
        switch (rn) {
#define CJX_A_CASE(R) \
  case R: k_colifft_window_reg<R><<<gc, kWarps * 32, sa_reg, stream>>>(hb, t1, g); break;
          CJX_A_CASE(1) CJX_A_CASE(2) CJX_A_CASE(3) CJX_A_CASE(4) CJX_A_CASE(5)
          CJX_A_CASE(6) CJX_A_CASE(8) CJX_A_CASE(10) CJX_A_CASE(12) CJX_A_CASE(16)
#undef CJX_A_CASE
        }
      } else {
        (g.plan_n.primes ? k_colifft_window<true> : k_colifft_window<false>)<<<gc, kWarps * 32, sa, stream>>>(hb, t1,
                                                                                                             g);
      }
      prof_end("k_colifft_window", stream);
    } else {
      const dim3 ga((g.nxh + kWarps - 1) / kWarps, cnt);
      prof_begin(stream);
      const bool bricked = (g.flags & CJX_GRID_BRICKED) != 0;
#define CJX_GC(S)                                                                                     \
  if (bricked)                                                                                        \
    (g.plan_n.primes ? k_gather_colifft<S, BrickLayout, true> : k_gather_colifft<S, BrickLayout, false>)     \
        <<<ga, kWarps * 32, sa, stream>>>(grid, params, order, t1, g, k0);                              \
  else                                                                                                \
    (g.plan_n.primes ? k_gather_colifft<S, LinearLayout, true> : k_gather_colifft<S, LinearLayout, false>)   \
        <<<ga, kWarps * 32, sa, stream>>>(grid, params, order, t1, g, k0);
      if (ilp == 4) {
        CJX_GC(4)
      } else if (ilp == 2) {
        CJX_GC(2)
      } else {
        CJX_GC(1)
      }
#undef CJX_GC
      prof_end("k_gather_colifft", stream);
    }
  return check_cuda(cudaGetLastError(), "forward launch");
}

// The row pass for one chunk: T1 -> T2.
static int launch_rows(const SliceGeom& g, const float2* t1, float2* t2, int cnt, cudaStream_t stream,
                       const Tuning& tn) {
  if (g.flags & CJX_EWALD_SPHERE) return launch_ewald_rows(g, t1, t2, cnt, stream, tn);
  const int rn = reg_fft_radix(g.n), rpx = reg_fft_radix(g.px);
  const bool fast = tn.fft_mode >= 1;
  const size_t sb = smem_b(g);
  const size_t sb_reg =
      sizeof(float2) * (size_t)(g.n + g.px + kWarps * rows_stride(g.n, g.px, rn == 16)) + sizeof(int) * (size_t)g.px;
    prof_begin(stream);
    const dim3 gb((g.py + 2 * kWarps - 1) / (2 * kWarps), cnt);
    if (fast && rn && rpx) {
      switch (rn) {
#define CJX_B_CASE(R) \
  case R:                                                                                   \
    if (R == 16 && tn.fft_mode == 3)                                                        \
      k_rows_reg<16, true><<<gb, kWarps * 32, sb_reg, stream>>>(t1, t2, g, rpx);             \
    else                                                                                    \
      k_rows_reg<R><<<gb, kWarps * 32, sb_reg, stream>>>(t1, t2, g, rpx);                    \
    break;
        CJX_B_CASE(1) CJX_B_CASE(2) CJX_B_CASE(3) CJX_B_CASE(4) CJX_B_CASE(5)
        CJX_B_CASE(6) CJX_B_CASE(8) CJX_B_CASE(10) CJX_B_CASE(12) CJX_B_CASE(16)
#undef CJX_B_CASE
      }
    } else {
      (g.plan_n.primes || g.plan_px.primes ? k_rows_c2r_r2c<true> : k_rows_c2r_r2c<false>)<<<gb, kWarps * 32, sb,
                                                                                           stream>>>(t1, t2, g);
    }
    prof_end("k_rows_c2r_r2c", stream);
  return check_cuda(cudaGetLastError(), "forward launch");
}

// Passes up to T2 (gather, column inverse FFT + window, rows) for one chunk of
// `cnt` images starting at processing index k0.
int launch_forward_to_t2(const SliceGeom& g, const float2* grid, const cjx_image_params* params, const int32_t* order,
                         int64_t k0, int cnt, float2* t1, float2* t2, float2* hb, cudaStream_t stream,
                         const Tuning& tn) {
  if (int e = launch_front(g, grid, params, order, k0, cnt, t1, hb, stream, tn)) return e;
  return launch_rows(g, t1, t2, cnt, stream, tn);
}

Tuning current_tuning() {
  return Tuning{(int)g_gather_ilp.load(), (int)g_gather_tile.load(), (int)g_gather_mode.load(),
                (int)g_fft_mode.load(), (int)g_scatter_vec.load(), (int)g_spline_ilp.load(),
                (int)g_multi_waves.load()};
}

// The last pass for one chunk: column FFT + scale, CTF, envelope, translation (and filter), T2 -> out.
static int launch_tail(const SliceGeom& g, const float2* t2, const cjx_image_params* params, const int32_t* order,
                       float2* out, int64_t k0, int cnt, cudaStream_t stream, const Tuning& tn) {
  if (g.flags & CJX_EWALD_SPHERE) return launch_ewald_colfft(g, t2, params, order, out, k0, cnt, stream, tn);
  const float norm = (float)(1.0 / ((double)g.n * (double)g.n));
  const int rpy = reg_fft_radix(g.py);
  const size_t sc = smem_c(g);
  const size_t sc_reg = sizeof(float2) * (size_t)(2 * g.py + kWarps * (stage_r_size(rpy) + 1));
  prof_begin(stream);
  const dim3 gcc((g.pxh + kWarps - 1) / kWarps, cnt);
  if (tn.fft_mode >= 1 && rpy) {
    switch (rpy) {
#define CJX_C_CASE(R) \
  case R:             \
    k_colfft_epilogue_reg<R><<<gcc, kWarps * 32, sc_reg, stream>>>(t2, params, order, out, g, k0, norm); break;
      CJX_C_CASE(1) CJX_C_CASE(2) CJX_C_CASE(3) CJX_C_CASE(4) CJX_C_CASE(5)
      CJX_C_CASE(6) CJX_C_CASE(8) CJX_C_CASE(10) CJX_C_CASE(12) CJX_C_CASE(16)
#undef CJX_C_CASE
    }
  } else {
    (g.plan_py.primes ? k_colfft_epilogue<true> : k_colfft_epilogue<false>)<<<gcc, kWarps * 32, sc, stream>>>(
        t2, params, order, out, g, k0, norm);
  }
  prof_end("k_colfft_epilogue", stream);
  return check_cuda(cudaGetLastError(), "forward launch");
}

int launch_forward(const SliceGeom& g, const float2* grid, const cjx_image_params* params, const int32_t* order,
                   int64_t n_images, float2* out, void* workspace, int64_t chunk, cudaStream_t stream,
                   const Tuning& tn) {
  if (n_images == 0) return CJX_OK;
  if (!needs_resize(g) && (g.flags & CJX_EWALD_SPHERE))
    return launch_ewald_direct(g, grid, params, order, n_images, out, stream);
  if (!needs_resize(g)) {
    const int total = g.n * g.nxh;
    const int blocks = std::min((total + 255) / 256, 1024);
    for (int64_t k0 = 0; k0 < n_images; k0 += 65535) {
      const int cnt = (int)std::min<int64_t>(65535, n_images - k0);
      prof_begin(stream);
      if ((g.flags & CJX_GRID_SPLINE) && (g.flags & CJX_GRID_BRICKED_PAIRS))
        k_slice_direct<SplinePairLayout><<<dim3(blocks, cnt), 256, 0, stream>>>(grid, params, order, out, g, k0);
      else if ((g.flags & CJX_GRID_SPLINE) && (g.flags & CJX_GRID_BRICKED))
        k_slice_direct<SplineBrickLayout><<<dim3(blocks, cnt), 256, 0, stream>>>(grid, params, order, out, g, k0);
      else if (g.flags & CJX_GRID_SPLINE)
        k_slice_direct<SplineLinearLayout><<<dim3(blocks, cnt), 256, 0, stream>>>(grid, params, order, out, g, k0);
      else if (g.flags & CJX_GRID_BRICKED_PAIRS)
        k_slice_direct<PairLayout><<<dim3(blocks, cnt), 256, 0, stream>>>(grid, params, order, out, g, k0);
      else if (g.flags & CJX_GRID_BRICKED)
        k_slice_direct<BrickLayout><<<dim3(blocks, cnt), 256, 0, stream>>>(grid, params, order, out, g, k0);
      else
        k_slice_direct<LinearLayout><<<dim3(blocks, cnt), 256, 0, stream>>>(grid, params, order, out, g, k0);
      prof_end("k_slice_direct", stream);
    }
    return check_cuda(cudaGetLastError(), "k_slice_direct launch");
  }
  if (int e = ensure_smem_attrs()) return e;
  const size_t sa = smem_a(g), sb = smem_b(g), sc = smem_c(g);
  if (sa > 227 * 1024 || sb > 227 * 1024 || sc > 227 * 1024)
    return fail(CJX_ERR_UNSUPPORTED, "shared-memory footprint exceeds 227 KB for these sizes");
  float2* t1 = static_cast<float2*>(workspace);
  float2* t2 = t1 + (size_t)chunk * g.py * g.ld1;
  float2* hb = t2 + (size_t)chunk * g.py * g.ld2;
  for (int64_t k0 = 0; k0 < n_images; k0 += chunk) {
    const int cnt = (int)std::min<int64_t>(chunk, n_images - k0);
    if (int e = launch_forward_to_t2(g, grid, params, order, k0, cnt, t1, t2, hb, stream, tn)) return e;
    if (int e = launch_tail(g, t2, params, order, out, k0, cnt, stream, tn)) return e;
  }
  return check_cuda(cudaGetLastError(), "forward launch");
}

// ---------------------------------------------------------------------------
// Mixed-size batches in waves: one launch per pass for all groups
// ---------------------------------------------------------------------------
size_t front_wave_smem(const SliceGeom& g);
int front_wave_ctas_per_image(const SliceGeom& g);
int launch_front_wave(const Wave& w, int ctas, size_t smem, cudaStream_t stream);

// A group can join the waves when it takes the fused register-FFT path end to
// end: trilinear slice (not spline, not Ewald), resize path, N, Py, Px of the
// register-FFT sizes, no fused filter, and the same grid layout as the others.
bool wave_eligible(const SliceGeom& g, const Tuning& tn) {
  return needs_resize(g) && !(g.flags & (CJX_GRID_SPLINE | CJX_EWALD_SPHERE)) && !g.filter &&
         tn.fft_mode >= 1 && tn.gather_mode == 2 && reg_fft_radix(g.n) && reg_fft_radix(g.py) &&
         reg_fft_radix(g.px);
}

size_t wave_bytes_per_image(const SliceGeom& g) {
  return sizeof(float2) * ((size_t)g.py * g.ld1 + (size_t)g.py * g.ld2);
}

// Number of waves whose slices fit the workspace (images per wave of group i
// in per_wave[i]), or 0 when even one image of every group does not fit (the
// groups then run one after another).  More waves never help beyond the
// largest group's image count, where every slice is one image.
int64_t plan_waves(const WaveInput* in, int n_in, size_t workspace_bytes, int64_t* per_wave) {
  double total = 0.0;
  int64_t n_max = 0;
  for (int i = 0; i < n_in; ++i) {
    total += (double)in[i].n * (double)wave_bytes_per_image(in[i].g);
    n_max = std::max<int64_t>(n_max, in[i].n);
  }
  if (n_max == 0) return 0;
  for (int64_t waves = std::max<int64_t>(1, (int64_t)std::ceil(total / (double)workspace_bytes)); waves <= n_max;
       ++waves) {
    size_t need = 0;
    for (int i = 0; i < n_in; ++i) {
      per_wave[i] = (in[i].n + waves - 1) / waves;
      need += (size_t)per_wave[i] * wave_bytes_per_image(in[i].g);
    }
    if (need <= workspace_bytes) return waves;
  }
  return 0;
}

// Every group's images in waves that fit the workspace: wave v holds images
// [v c_i, (v + 1) c_i) of group i (c_i = ceil(n_i / waves)), so all groups end
// together; per wave the front, row and column passes are one launch each,
// the CTAs of the groups one after another in each launch.
int launch_forward_waves(const WaveInput* in, int n_in, void* workspace, size_t workspace_bytes, cudaStream_t stream,
                         const Tuning& tn) {
  if (n_in < 1 || n_in > kMaxWaveGroups) return fail(CJX_ERR_UNSUPPORTED, "waves take 1 to 8 groups");
  if (int e = ensure_smem_attrs()) return e;
  static PerDeviceOnce once;
  const cudaError_t ea = once.run([] {
    // the kernels also hold static shared tables, so the dynamic limit stays below 227 KB
    cudaError_t e = cudaFuncSetAttribute(k_rows_wave, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_tail_wave, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    return e;
  });
  if (ea != cudaSuccess) return check_cuda(ea, "cudaFuncSetAttribute (wave passes)");
  int64_t n_max = 0;
  size_t s_front = 0, s_rows = 0, s_tail = 0;
  for (int i = 0; i < n_in; ++i) {
    const SliceGeom& g = in[i].g;
    n_max = std::max<int64_t>(n_max, in[i].n);
    s_front = std::max(s_front, front_wave_smem(g));
    s_rows = std::max(s_rows, sizeof(float2) * (size_t)(g.n + g.px + kWarps * rows_stride(g.n, g.px, reg_fft_radix(g.n) == 16)) +
                                  sizeof(int) * (size_t)g.px);
    s_tail = std::max(s_tail, sizeof(float2) * (size_t)(2 * g.py + kWarps * (stage_r_size(reg_fft_radix(g.py)) + 1)));
  }
  if (n_max == 0) return CJX_OK;
  std::vector<int64_t> per_wave(n_in);
  const int64_t waves = plan_waves(in, n_in, workspace_bytes, per_wave.data());
  if (waves <= 0) return fail(CJX_ERR_WORKSPACE, "workspace smaller than one image of every group");
  Wave w{};
  w.n = n_in;
  w.t512 = tn.fft_mode >= 2;
  w.rows_t512 = tn.fft_mode == 3;
  char* base = static_cast<char*>(workspace);
  for (int i = 0; i < n_in; ++i) {
    WaveGroup& q = w.grp[i];
    q.g = in[i].g;
    q.grid = in[i].grid;
    q.params = in[i].params;
    q.order = in[i].order;
    q.out = in[i].out;
    q.t1 = reinterpret_cast<float2*>(base);
    q.t2 = q.t1 + (size_t)per_wave[i] * q.g.py * q.g.ld1;
    base += (size_t)per_wave[i] * wave_bytes_per_image(q.g);
  }
  for (int64_t v = 0; v < waves; ++v) {
    int64_t ctas[3] = {0, 0, 0};
    for (int i = 0; i < n_in; ++i) {
      WaveGroup& q = w.grp[i];
      q.k0 = std::min<int64_t>(v * per_wave[i], in[i].n);
      q.cnt = (int)std::min<int64_t>(per_wave[i], in[i].n - q.k0);
      const int64_t per[3] = {front_wave_ctas_per_image(q.g), (q.g.py + 2 * kWarps - 1) / (2 * kWarps),
                              (q.g.pxh + kWarps - 1) / kWarps};
      for (int p = 0; p < 3; ++p) {
        q.cta0[p] = (int)ctas[p];
        ctas[p] += per[p] * q.cnt;
      }
    }
    if (ctas[0] == 0) continue;
    if (ctas[0] > 2147483647LL || ctas[1] > 2147483647LL || ctas[2] > 2147483647LL)
      return fail(CJX_ERR_UNSUPPORTED, "too many CTAs in one wave");
    if (int e = launch_front_wave(w, (int)ctas[0], s_front, stream)) return e;
    prof_begin(stream);
    k_rows_wave<<<(unsigned)ctas[1], kWarps * 32, s_rows, stream>>>(w);
    prof_end("k_rows_wave", stream);
    prof_begin(stream);
    k_tail_wave<<<(unsigned)ctas[2], kWarps * 32, s_tail, stream>>>(w);
    prof_end("k_tail_wave", stream);
    if (int e = check_cuda(cudaGetLastError(), "wave launch")) return e;
  }
  return CJX_OK;
}

// ---------------------------------------------------------------------------
// Volume re-layout: C-order [z][y][x] -> BrickLayout (one-time preparation).
// One thread per bricked element; elements beyond N on any axis are zero.
// ---------------------------------------------------------------------------
__global__ void k_brick_volume(const float2* __restrict__ grid, float2* __restrict__ bricked, int n, int nb) {
  const int64_t total = (int64_t)nb * nb * nb * 512;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int w = (int)(e & 511);
    const int64_t blk = e >> 9;
    const int bx = (int)(blk % nb), by = (int)((blk / nb) % nb), bz = (int)(blk / ((int64_t)nb * nb));
    // de-interleave the Morton index (x bits 0,3,6; y bits 1,4,7; z bits 2,5,8)
    const int x = bx * 8 + ((w & 1) | ((w >> 2) & 2) | ((w >> 4) & 4));
    const int y = by * 8 + (((w >> 1) & 1) | ((w >> 3) & 2) | ((w >> 5) & 4));
    const int z = bz * 8 + (((w >> 2) & 1) | ((w >> 4) & 2) | ((w >> 6) & 4));
    bricked[e] = (x < n && y < n && z < n) ? grid[((int64_t)z * n + y) * n + x] : make_float2(0.f, 0.f);
  }
}

// x-pair entries (g(x), g(x + 1)) in the same bricked order; 0 beyond the volume.
__global__ void k_brick_volume_pairs(const float2* __restrict__ grid, float4* __restrict__ out, int n, int nb) {
  const int64_t total = (int64_t)nb * nb * nb * 512;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int w = (int)(e & 511);
    const int64_t blk = e >> 9;
    const int bx = (int)(blk % nb), by = (int)((blk / nb) % nb), bz = (int)(blk / ((int64_t)nb * nb));
    const int x = bx * 8 + ((w & 1) | ((w >> 2) & 2) | ((w >> 4) & 4));
    const int y = by * 8 + (((w >> 1) & 1) | ((w >> 3) & 2) | ((w >> 5) & 4));
    const int z = bz * 8 + (((w >> 2) & 1) | ((w >> 4) & 2) | ((w >> 6) & 4));
    float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
    if (y < n && z < n) {
      const int64_t row = ((int64_t)z * n + y) * n;
      if (x < n) a = grid[row + x];
      if (x + 1 < n) b = grid[row + x + 1];
    }
    out[e] = make_float4(a.x, a.y, b.x, b.y);
  }
}

int launch_brick_volume_pairs(int n, const float2* grid, float4* out, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  prof_begin(stream);
  k_brick_volume_pairs<<<sms * 8, 256, 0, stream>>>(grid, out, n, brick_blocks(n));
  prof_end("k_brick_volume_pairs", stream);
  return check_cuda(cudaGetLastError(), "k_brick_volume_pairs launch");
}

size_t bricked_elements(int n) {
  const size_t nb = (size_t)brick_blocks(n);
  return nb * nb * nb * 512;
}

int launch_brick_volume(int n, const float2* grid, float2* bricked, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  prof_begin(stream);
  k_brick_volume<<<sms * 8, 256, 0, stream>>>(grid, bricked, n, brick_blocks(n));
  prof_end("k_brick_volume", stream);
  return check_cuda(cudaGetLastError(), "k_brick_volume launch");
}

// ---------------------------------------------------------------------------
// Read-bandwidth probe
// ---------------------------------------------------------------------------
__global__ void k_read_probe(const float4* __restrict__ buf, size_t n16, int passes, float* sink) {
  float acc = 0.f;
  for (int p = 0; p < passes; ++p) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x) {
      const float4 v = __ldcg(&buf[i]);
      acc += (v.x + v.y) + (v.z + v.w);
    }
  }
  if (acc == 1.2345e-30f) sink[0] = acc;  // keeps the loads live
}

int launch_read_probe(const void* buf, size_t bytes, int passes, void* sink, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  prof_begin(stream);
  k_read_probe<<<sms * 4, 512, 0, stream>>>(static_cast<const float4*>(buf), bytes / 16, passes,
                                            static_cast<float*>(sink));
  prof_end("k_read_probe", stream);
  return check_cuda(cudaGetLastError(), "k_read_probe launch");
}

}  // namespace cjx
