// fine.cu -- the per-pixel kernels of the fine stage (python/optflow_ref/phaseflow.py:427-511,
// rust/crates/optflow-core/src/phaseflow.rs:1514-1613): smoothing, splines, warp, accumulate, window moments
// and the local solve, the energy median, the confidence and the trusted pre-warp.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "kernels.cuh"

#include <cooperative_groups.h>
#include <cuda_pipeline.h>

namespace ofc {

// ---------------------------------------------------------------- separable correlation ("nearest")
template <class Tin>
__global__ void k_corr_y(const Tin* __restrict__ in, double* __restrict__ out, int W, int H,
                         const double* __restrict__ taps, int r) {
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  int pl = blockIdx.z;
  if (x >= W) return;
  const Tin* a = in + (size_t)pl * W * H;
  double s = 0;
  for (int j = -r; j <= r; j++) {
    int yy = min(max(y + j, 0), H - 1);
    s += taps[j + r] * (double)a[(size_t)yy * W + x];
  }
  out[(size_t)pl * W * H + (size_t)y * W + x] = s;
}

__global__ void k_corr_x(const double* __restrict__ in, double* __restrict__ out, int W, int H,
                         const double* __restrict__ taps, int r) {
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  int pl = blockIdx.z;
  if (x >= W) return;
  const double* a = in + (size_t)pl * W * H + (size_t)y * W;
  double s = 0;
  for (int j = -r; j <= r; j++) {
    int xx = min(max(x + j, 0), W - 1);
    s += taps[j + r] * a[xx];
  }
  out[(size_t)pl * W * H + (size_t)y * W + x] = s;
}

// The same correlations for the default smoothing window (r = 16, sigma_s = 4). y: a thread owns CY_RY
// consecutive rows of a column and loads their 2r + CY_RY input rows once (instead of 2r + 1 loads per output,
// most of them L2 traffic); x: a block stages a row segment and its halo in shared memory and a thread forms
// CX_RX consecutive outputs from one register window (odd CX_RX: the warp's reads fall on distinct banks).
// Symmetric taps are paired (k(t) = k(-t)). Eight rows per thread in y (40 loads for 8 outputs, 80 registers, six
// blocks per SM) took 0.040 ms per pass of the two field planes at 2048^2 against 0.052 ms with four.
constexpr int CORR_R = 16, CY_RY = 8, CX_RX = 3;

__global__ void __launch_bounds__(128, 6) k_corr_y_rb(const double* __restrict__ in, double* __restrict__ out, int W,
                                                     int H, const double* __restrict__ taps) {
  grid_dep_wait();
  constexpr int R = CORR_R, RY = CY_RY, NV = RY + 2 * R;
  __shared__ double tk[R + 1];
  if (threadIdx.x <= R) tk[threadIdx.x] = taps[R + threadIdx.x];
  __syncthreads();
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y0 = blockIdx.y * RY;
  if (x >= W) return;
  const double* a = in + (size_t)blockIdx.z * W * H + x;
  double v[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) v[i] = a[(size_t)min(max(y0 - R + i, 0), H - 1) * W];
  double acc[RY];
#pragma unroll
  for (int j = 0; j < RY; j++) acc[j] = tk[0] * v[j + R];
#pragma unroll
  for (int t = 1; t <= R; t++) {
    const double k = tk[t];
#pragma unroll
    for (int j = 0; j < RY; j++) acc[j] = fma(k, v[j + R + t] + v[j + R - t], acc[j]);
  }
  double* o = out + (size_t)blockIdx.z * W * H + x;
#pragma unroll
  for (int j = 0; j < RY; j++)
    if (y0 + j < H) o[(size_t)(y0 + j) * W] = acc[j];
}

__global__ void __launch_bounds__(128) k_corr_x_rb(const double* __restrict__ in, double* __restrict__ out, int W, int H,
                                                  const double* __restrict__ taps) {
  grid_dep_wait();
  constexpr int R = CORR_R, RX = CX_RX, NT = 128, SEG = NT * RX, WIN = SEG + 2 * R, NV = RX + 2 * R;
  __shared__ double tk[R + 1];
  __shared__ double wb[WIN];
  __shared__ double ob[SEG];
  const int tid = threadIdx.x, x0 = blockIdx.x * SEG;
  const double* row = in + (size_t)blockIdx.z * W * H + (size_t)blockIdx.y * W;
  if (tid <= R) tk[tid] = taps[R + tid];
  for (int i = tid; i < WIN; i += NT) wb[i] = row[min(max(x0 - R + i, 0), W - 1)];
  __syncthreads();
  double v[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) v[i] = wb[tid * RX + i];
  double acc[RX];
#pragma unroll
  for (int j = 0; j < RX; j++) acc[j] = tk[0] * v[j + R];
#pragma unroll
  for (int t = 1; t <= R; t++) {
    const double k = tk[t];
#pragma unroll
    for (int j = 0; j < RX; j++) acc[j] = fma(k, v[j + R + t] + v[j + R - t], acc[j]);
  }
#pragma unroll
  for (int j = 0; j < RX; j++) ob[tid * RX + j] = acc[j];
  __syncthreads();
  double* o = out + (size_t)blockIdx.z * W * H + (size_t)blockIdx.y * W;
  for (int i = tid; i < SEG; i += NT)
    if (x0 + i < W) o[x0 + i] = ob[i];
}

void launch_corr_y(const double* in, double* out, int n_planes, int W, int H, const double* taps, int r, cudaStream_t st) {
  if (r == CORR_R) {
    dim3 g(div_up(W, 128), div_up(H, CY_RY), n_planes);
    OFC_LAUNCH_PDL(k_corr_y_rb, g, 128, 0, st, in, out, W, H, taps);
    return;
  }
  dim3 g(div_up(W, 128), H, n_planes);
  OFC_LAUNCH(k_corr_y<double>, g, 128, 0, st, in, out, W, H, taps, r);
}
void launch_corr_x(const double* in, double* out, int n_planes, int W, int H, const double* taps, int r, cudaStream_t st) {
  if (r == CORR_R) {
    dim3 g(div_up(W, 128 * CX_RX), H, n_planes);
    OFC_LAUNCH_PDL(k_corr_x_rb, g, 128, 0, st, in, out, W, H, taps);
    return;
  }
  dim3 g(div_up(W, 128), H, n_planes);
  OFC_LAUNCH(k_corr_x, g, 128, 0, st, in, out, W, H, taps, r);
}
void launch_corr_y_f32in(const float* in, double* out, int W, int H, const double* taps, int r, cudaStream_t st) {
  dim3 g(div_up(W, 128), H, 1);
  OFC_LAUNCH(k_corr_y<float>, g, 128, 0, st, in, out, W, H, taps, r);
}

// ---------------------------------------------------------------- B-spline prefilter in global memory
// Segmented recursive filter along one axis (interp.py:13-27): a line of length n with element stride
// `es`, lines `ls` apart. Each thread filters one segment of one line, entering it after a warm-up of
// IIR_WARM samples (exact when the warm-up reaches the line's start/end). Causal: in -> y (times 6);
// anticausal: y -> out.
constexpr int SEG = 32;

template <class Tin>
__global__ void k_iir_causal(const Tin* __restrict__ in, double* __restrict__ y, int n, int nlines, long es, long ls,
                             long plane) {
  int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= nlines) return;
  const int s0 = blockIdx.y * SEG;
  if (s0 >= n) return;
  const int e0 = min(n, s0 + SEG);
  const Tin* a = in + (size_t)blockIdx.z * plane + (size_t)line * ls;
  double* o = y + (size_t)blockIdx.z * plane + (size_t)line * ls;
  if (n == 1) { o[0] = (double)a[0]; return; }
  const double z = bspline_z();
  double acc;
  int i0;
  if (s0 - IIR_WARM <= 0) {
    int hz = min(n, HORIZON);
    acc = 0;
    double zk = 1;
    for (int k = 0; k < hz; k++) { acc += zk * (6.0 * (double)a[(size_t)k * es]); zk *= z; }
    if (s0 == 0) o[0] = acc;
    for (int i = 1; i < s0; i++) acc = 6.0 * (double)a[(size_t)i * es] + z * acc;
    i0 = s0 == 0 ? 1 : s0;
  } else {
    acc = 0;
    for (int i = s0 - IIR_WARM; i < s0; i++) acc = 6.0 * (double)a[(size_t)i * es] + z * acc;
    i0 = s0;
  }
  for (int i = i0; i < e0; i++) {
    acc = 6.0 * (double)a[(size_t)i * es] + z * acc;
    o[(size_t)i * es] = acc;
  }
}

template <class Tout>
__global__ void k_iir_anticausal(const double* __restrict__ y, Tout* __restrict__ out, int n, int nlines, long es,
                                 long ls, long plane) {
  int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= nlines) return;
  const int s0 = blockIdx.y * SEG;
  if (s0 >= n) return;
  const int e0 = min(n, s0 + SEG);
  const double* a = y + (size_t)blockIdx.z * plane + (size_t)line * ls;
  Tout* o = out + (size_t)blockIdx.z * plane + (size_t)line * ls;
  if (n == 1) { o[0] = (Tout)a[0]; return; }
  const double z = bspline_z();
  const double g = z / (z * z - 1.0);
  double c;
  if (e0 + IIR_WARM >= n - 1) {
    c = g * (a[(size_t)(n - 1) * es] + z * a[(size_t)(n - 2) * es]);
    if (e0 == n) o[(size_t)(n - 1) * es] = (Tout)c;
    for (int i = n - 2; i >= e0; i--) c = z * (c - a[(size_t)i * es]);
    if (e0 == n) {
      for (int i = n - 2; i >= s0; i--) { c = z * (c - a[(size_t)i * es]); o[(size_t)i * es] = (Tout)c; }
      return;
    }
  } else {
    c = 0;
    for (int i = e0 + IIR_WARM; i >= e0; i--) c = z * (c - a[(size_t)i * es]);
  }
  // c = c[e0]
  for (int i = e0 - 1; i >= s0; i--) { c = z * (c - a[(size_t)i * es]); o[(size_t)i * es] = (Tout)c; }
}

// Both recursions along x (rows) in one pass through a shared-memory tile: a block of XR_ROWS threads owns
// XR_ROWS rows and the column segment [s0, s0 + XR_SEG); it loads columns [s0 - IIR_WARM, e0 + IIR_WARM]
// (clamped to the row) with coalesced row reads, each thread runs the causal recursion over its tile row (warm-up
// from the tile's start, or the exact start at column 0) and then the anticausal one down to s0 (warm-up from the
// tile's end, or the exact start at the row's end), and the block stores the segment with coalesced row writes.
// One thread per row makes the recursion sequential in a row; an odd row stride keeps the threads' column
// accesses on distinct banks.
constexpr int XR_ROWS = 64, XR_SEG = 64, XR_TW = XR_SEG + 2 * IIR_WARM + 1;  // 121 doubles per tile row (odd)

// ILV: the planes (two) are written interleaved, out[2 p + plane]
template <class Tout, bool ILV>
__global__ void __launch_bounds__(XR_ROWS) k_iir_x(const double* __restrict__ in, Tout* __restrict__ out, int n, int nrows,
                                                  long plane) {
  extern __shared__ double tile[];  // XR_ROWS x XR_TW
  const int r0 = blockIdx.y * XR_ROWS, s0 = blockIdx.x * XR_SEG;
  const int e0 = min(n, s0 + XR_SEG), c0 = max(0, s0 - IIR_WARM), c1 = min(n, e0 + IIR_WARM + 1), cw = c1 - c0;
  const double* a = in + (size_t)blockIdx.z * plane;
  Tout* o = out + (size_t)blockIdx.z * plane;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  // asynchronous copies: the whole tile is in flight at once (a load-then-store loop waits a DRAM latency per row)
  for (int rr = wid; rr < XR_ROWS; rr += nw) {
    if (r0 + rr >= nrows) break;
    const double* src = a + (size_t)(r0 + rr) * n + c0;
    for (int c = lane; c < cw; c += 32) __pipeline_memcpy_async(&tile[rr * XR_TW + c], src + c, sizeof(double));
  }
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
  const int row = threadIdx.x;
  if (r0 + row < nrows) {
    double* t = tile + row * XR_TW;  // t[i - c0] = value at column i
    if (n == 1) {
      // a single column: the coefficient is the value (as the separate passes give)
    } else {
      const double z = bspline_z();
      double acc;
      int i0;
      if (c0 == 0) {  // exact start: y[0] = sum_{k < min(n, 21)} z^k 6 x[k]
        const int hz = min(n, HORIZON);
        acc = 0;
        double zk = 1;
        for (int k = 0; k < hz; k++) {
          acc += zk * (6.0 * t[k]);
          zk *= z;
        }
        t[0] = acc;
        i0 = 1;
      } else {
        acc = 0;
        i0 = 0;
      }
#pragma unroll 4
      for (int i = i0; i < cw; i++) {
        acc = 6.0 * t[i] + z * acc;
        t[i] = acc;
      }
      const double g = z / (z * z - 1.0);
      double c;
      int i1;
      if (c1 == n) {  // exact start: c[n-1] = z / (z^2 - 1) (y[n-1] + z y[n-2])
        c = g * (t[cw - 1] + z * t[cw - 2]);
        t[cw - 1] = c;
        i1 = cw - 2;
      } else {
        c = 0;
        i1 = cw - 1;
      }
#pragma unroll 4
      for (int i = i1; i >= s0 - c0; i--) {
        c = z * (c - t[i]);
        t[i] = c;
      }
    }
  }
  __syncthreads();
  for (int rr = wid; rr < XR_ROWS; rr += nw) {
    if (r0 + rr >= nrows) break;
    const double* t = tile + rr * XR_TW + (s0 - c0);
    if (ILV) {
      Tout* dst = out + ((size_t)(r0 + rr) * n + s0) * 2 + blockIdx.z;
      for (int c = lane; c < e0 - s0; c += 32) dst[2 * c] = (Tout)t[c];
    } else {
      Tout* dst = o + (size_t)(r0 + rr) * n + s0;
      for (int c = lane; c < e0 - s0; c += 32) dst[c] = (Tout)t[c];
    }
  }
}

// y pass: in -> tmp (causal) -> tmp2 (anticausal); x pass: tmp2 -> out (ILV: two planes interleaved). tmp may alias
// out (it is dead once the x pass starts); tmp2 must not, since the x pass's tiles overlap.
template <class Tin, class Tout, bool ILV = false>
static void bspline_axes(const Tin* in, Tout* out, double* tmp, double* tmp2, int n_planes, int W, int H, cudaStream_t st) {
  long plane = (long)W * H;
  // along y: lines = columns (stride 1 apart), element stride W
  dim3 gy(div_up(W, 128), div_up(H, SEG), n_planes);
  OFC_LAUNCH((k_iir_causal<Tin>), gy, 128, 0, st, in, tmp, H, W, (long)W, 1L, plane);
  OFC_LAUNCH((k_iir_anticausal<double>), gy, 128, 0, st, tmp, tmp2, H, W, (long)W, 1L, plane);
  // along x: both recursions in one pass through shared-memory tiles
  const size_t sm = (size_t)XR_ROWS * XR_TW * sizeof(double);
  raise_smem_limit((const void*)k_iir_x<Tout, ILV>, sm);
  dim3 gx(div_up(W, XR_SEG), div_up(H, XR_ROWS), n_planes);
  OFC_LAUNCH((k_iir_x<Tout, ILV>), gx, XR_ROWS, sm, st, tmp2, out, W, H, plane);
}

void launch_bspline_f64(const double* in, double* out, double* tmp, int n_planes, int W, int H, cudaStream_t st) {
  // out doubles as the causal scratch of the y pass; tmp holds the y pass's result for the x pass
  bspline_axes<double, double>(in, out, (double*)out, tmp, n_planes, W, H, st);
}

void launch_bspline_f64_pair(const double* in, double2* out, double* tmp, int W, int H, cudaStream_t st) {
  // out (2 W H doubles) doubles as the causal scratch of the y pass; tmp holds the y pass's result
  bspline_axes<double, double, true>(in, (double*)out, (double*)out, tmp, 2, W, H, st);
}

void launch_bspline_f32(const float* in, float* out, double* tmp, int W, int H, cudaStream_t st) {
  // tmp holds 2 planes
  bspline_axes<float, float>(in, out, tmp, tmp + (size_t)W * H, 1, W, H, st);
}

// ---------------------------------------------------------------- warp
__global__ void __launch_bounds__(128, 8) k_warp(const float* __restrict__ c2, int w2, int h2, const double* __restrict__ sx,
                       const double* __restrict__ sy, long shx, long shy, int W, int H, float* __restrict__ out) {
  grid_dep_wait();
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= W) return;
  for (int y = blockIdx.y; y < H; y += gridDim.y) {  // rows beyond the grid's 65535 in steps of gridDim.y
    size_t p = (size_t)y * W + x;
    Taps t;
    double v;
    if (make_taps(((double)x + (double)shx) + sx[p], ((double)y + (double)shy) + sy[p], w2, h2, t))
      v = sample_real(c2, w2, t);
    else
      v = nan("");
    out[p] = (float)v;
  }
}

// the warp as a plain gather: the form for coefficient planes whose row pitch is not a multiple of 16 bytes (no
// tensor map), and the reference the TMA-staged warp (warp_tma.cu) is checked against
void launch_warp_gather(const float* c2, int w2, int h2, const double* sx, const double* sy, long shx, long shy, int W,
                        int H, float* out, cudaStream_t st) {
  dim3 g(div_up(W, 128), (unsigned)std::min(H, 65535));
  OFC_LAUNCH_PDL(k_warp, g, 128, 0, st, c2, w2, h2, sx, sy, shx, shy, W, H, out);
}

// ---------------------------------------------------------------- accumulate
// One pixel per thread. The fixed point X' + s(X') = X + u(X) and the positions are float64; the responses are
// sampled with float32 weights and accumulation (they are stored as complex float32), and the phase difference
// angle(r1 conj(r2)) is taken in float32 by atan2_phase (the inputs carry float32 precision; the angle is within
// 5e-7 rad of theirs); c = dphi + gx u + gy v and the seven sums are float64, since u reaches tens of pixels and the
// residual sum gcc - theta . b cancels. |r1| |r2| is one square root of |r1|^2 |r2|^2, with |r1|^2 formed from the
// pack; the field spline is stored interleaved (one 16-byte load per tap for both components); the responses are
// stored in filter pairs, node-major, so one 16-byte load per tap serves two filters (96 tap loads per pixel at F = 12
// instead of 192).
// What bounds it is L1: the response taps, their prefetches and the ring keep it at 90 % of its throughput (DRAM at 43 %,
// issue at 50 %). 0.470 ms per launch in a 2048^2 pair, F = 12 (0.572 before the three steps below, the same sums bit for
// bit). The forms, one built beside the other, by python -m optflow_b200.measure accumulate (2048^2, the kernel repeated on
// one input): 0.433 ms as it is, and
//   - the reference pack by asynchronous copies into a ring of two filter pairs: a ring of three pairs 0.452, all of the
//     pairs staged at once 0.484 (24 KB per block instead of 8 leave L1 less room for the taps of the resident blocks);
//   - the taps' float32 sums and the two filters' atan polynomials in packed instructions (fma.rn.f32x2: two values per
//     issue slot, each rounded as by fmaf), the quotient of atan2 without a call, and the positions whose taps would mirror
//     or clamp (at the plane's border) out of line, so that the rest tests its range once;
//   - 32 x 4 pixels per block, 7 blocks per SM at 72 registers: 8 blocks at 64 registers 0.457, 6 at 80 0.459, 32 x 8 pixels
//     at 4 blocks 0.456;
//   - the next pair's tap rows prefetched into L1: 0.479 without.
// Slower, and not kept: two pixels of a column per thread sharing their tap rows (L1 wavefronts fall by a third, but
// 128 registers leave 16 warps per SM: 0.66 ms in the pair); the fixed point in a kernel of its own (0.122 + 0.424 ms: its
// loads no longer overlap the sums' arithmetic).
constexpr int ACC_BX = 32, ACC_BY = 4, ACC_T = ACC_BX * ACC_BY, ACC_MINB = 7;
constexpr int ACC_ST = 2;       // filter pairs in the ring of the reference pack
constexpr int ACC_MAXF = 56;    // the filters an earlier form held in shared memory at once; more stay refused

// the taps of a position at least one node inside the plane in both directions (no clamp, no reflection: what make_taps
// gives there); false elsewhere and for NaN
__device__ __forceinline__ bool taps_inside(double x, double y, int w, int h, int& node, double (&wx)[4], double (&wy)[4]) {
  if (!(x >= 1.0 && x < (double)(w - 2) && y >= 1.0 && y < (double)(h - 2))) return false;
  const double fx = floor(x), fy = floor(y);
  node = ((int)fy - 1) * w + ((int)fx - 1);
  bspline_weights(x - fx, wx);
  bspline_weights(y - fy, wy);
  return true;
}

// the field spline at (x, y) by the general taps
__device__ __noinline__ double2 field_general(const double2* __restrict__ cs, int W, int H, double x, double y) {
  Taps t;
  if (!make_taps(x, y, W, H, t)) return make_double2(nan(""), nan(""));
  return sample_pair(cs, W, t);
}

// the contributions of filters of phase difference dphi to a pixel's seven sums, from a filter's pack r1 (re, im, gx, gy)
// and its complex response sample b at X' (r2 of phaseflow.py:476-483)
__device__ __forceinline__ void acc_add(double (&a)[7], float4 r1, float br, float bi, float dph, double u, double v) {
  // |r1|^2 as the reference pack's amplitude squared (phaseflow.py:111), from the stored float32 response
  const float q1 = fmaf(r1.x, r1.x, fmaf(r1.y, r1.y, 1e-12f));
  const double dphi = (double)dph;
  const double wk = (double)sqrtf(q1 * fmaf(br, br, bi * bi));  // |r1| |r2|
  const double gx = r1.z, gy = r1.w;
  const double c = dphi + gx * u + gy * v;
  const double wgx = wk * gx, wgy = wk * gy;
  a[0] = fma(wgx, gx, a[0]);
  a[1] = fma(wgx, gy, a[1]);
  a[2] = fma(wgy, gy, a[2]);
  a[3] = fma(wgx, c, a[3]);
  a[4] = fma(wgy, c, a[4]);
  a[5] = fma(wk * c, c, a[5]);
  a[6] += wk;
}
// r1 conj(r2)
__device__ __forceinline__ void acc_cross(float4 r1, float br, float bi, float& im, float& re) {
  re = fmaf(r1.x, br, r1.y * bi);
  im = fmaf(r1.y, br, -r1.x * bi);
}

// a pixel whose taps mirror at the padded plane's border, or whose position is NaN: the general taps, from the pack in
// global memory
__device__ __noinline__ void acc_general(const float4* __restrict__ ref4, const float4* __restrict__ R4, int F, int ph,
                                         int pw, size_t N, size_t p, double px, double py, double u, double v,
                                         double* __restrict__ sums) {
  const float fnan = __int_as_float(0x7fc00000);
  const size_t plane = (size_t)ph * pw;
  double a[7] = {0, 0, 0, 0, 0, 0, 0};
  Taps t;
  const bool ok = make_taps(px + PAD, py + PAD, pw, ph, t);
#pragma unroll 1
  for (int k = 0; k < F; k++) {
    float br = fnan, bi = fnan;
    if (ok) {
      br = bi = 0.f;
      const float2* Rk = (const float2*)(R4 + (size_t)(k >> 1) * plane) + (k & 1);
#pragma unroll 1
      for (int jj = 0; jj < 4; jj++) {
        float ar = 0.f, ai = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float2 cv = __ldg(Rk + 2 * ((size_t)t.yi[jj] * pw + t.xi[q]));
          ar = fmaf((float)t.wx[q], cv.x, ar);
          ai = fmaf((float)t.wx[q], cv.y, ai);
        }
        br = fmaf((float)t.wy[jj], ar, br);
        bi = fmaf((float)t.wy[jj], ai, bi);
      }
    }
    const float4 r1 = __ldg(ref4 + (size_t)k * N + p);
    float im, re;
    acc_cross(r1, br, bi, im, re);
    acc_add(a, r1, br, bi, atan2_phase(im, re), u, v);
  }
#pragma unroll
  for (int i = 0; i < 7; i++) sums[i * N + p] = a[i];
}

__global__ void __launch_bounds__(ACC_T, ACC_MINB) k_accumulate(const float4* __restrict__ ref4, const float4* __restrict__ R4,
                                                      int F, int ph, int pw, const double* __restrict__ ux,
                                                      const double* __restrict__ uy, const double* __restrict__ sx,
                                                      const double* __restrict__ sy, const double2* __restrict__ cs,
                                                      int W, int H, double* __restrict__ sums) {
  grid_dep_wait();
  extern __shared__ float4 pk[];  // ACC_ST x 2 x ACC_T
  // a block covers ACC_BX x ACC_BY pixels: its warps' response taps share rows in L1
  const int x = blockIdx.x * ACC_BX + threadIdx.x, y = blockIdx.y * ACC_BY + threadIdx.y;
  const int tid = threadIdx.y * ACC_BX + threadIdx.x;
  if (x >= W || y >= H) return;
  const size_t N = (size_t)W * H;
  const size_t p = (size_t)y * W + x;
  // the reference pack of filter pair j into its slot of the ring (one group of asynchronous copies; an empty group
  // past the end)
  auto fetch = [&](int j) {
#pragma unroll
    for (int c = 0; c < 2; c++)
      if (2 * j + c < F)
        __pipeline_memcpy_async(&pk[((j % ACC_ST) * 2 + c) * ACC_T + tid], ref4 + (size_t)(2 * j + c) * N + p, 16);
    __pipeline_commit();
  };
#pragma unroll
  for (int j = 0; j < ACC_ST - 1; j++) fetch(j);
  const double u = ux[p], v = uy[p];
  const double tx = x + u, ty = y + v;
  double px = tx - sx[p], py = ty - sy[p];
  int base;
  double dwx[4], dwy[4];
  // X' + s(X') = X + u(X): two fixed-point steps on the spline of s (phaseflow.py:469-472)
#pragma unroll 1
  for (int it = 0; it < 2; it++) {
    double o1 = 0, o2 = 0;
    if (taps_inside(px, py, W, H, base, dwx, dwy)) {
      const double2* row = cs + base;
#pragma unroll
      for (int j = 0; j < 4; j++, row += W) {
        const double2 c0 = __ldg(row);
        double a1 = dwx[0] * c0.x, a2 = dwx[0] * c0.y;
#pragma unroll
        for (int k = 1; k < 4; k++) {
          const double2 cv = __ldg(row + k);
          a1 += dwx[k] * cv.x;
          a2 += dwx[k] * cv.y;
        }
        o1 += dwy[j] * a1;
        o2 += dwy[j] * a2;
      }
    } else {
      const double2 sv = field_general(cs, W, H, px, py);
      o1 = sv.x;
      o2 = sv.y;
    }
    px = tx - o1;
    py = ty - o2;
  }
  if (!taps_inside(px + PAD, py + PAD, pw, ph, base, dwx, dwy)) {
    __pipeline_wait_prior(0);
    acc_general(ref4, R4, F, ph, pw, N, p, px, py, u, v, sums);
    return;
  }
  unsigned long long wx[4], wy[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float a = (float)dwx[k], b = (float)dwy[k];
    wx[k] = f32x2(a, a);
    wy[k] = f32x2(b, b);
  }
  double a[7] = {0, 0, 0, 0, 0, 0, 0};
  const size_t plane = (size_t)ph * pw;
  // the responses in filter pairs, node-major: one 16-byte load per tap gives both filters of a pair; the taps are a
  // block (one address per row, the four loads at fixed offsets from it)
  const ulonglong2* Rj = reinterpret_cast<const ulonglong2*>(R4) + base;
  const int npairs = (F + 1) >> 1;
#pragma unroll 1
  for (int j = 0; j < npairs; j++, Rj += plane) {
    // the next pair's tap rows go into L1 meanwhile
    if (j + 1 < npairs) {
#pragma unroll
      for (int r = 0; r < 4; r++) asm volatile("prefetch.global.L1 [%0];" ::"l"(Rj + plane + r * pw));
    }
    unsigned long long s0 = 0ull, s1 = 0ull;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      unsigned long long r0 = 0ull, r1 = 0ull;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const ulonglong2 c = __ldg(Rj + (r * pw + q));
        r0 = fma_f32x2(wx[q], c.x, r0);
        r1 = fma_f32x2(wx[q], c.y, r1);
      }
      s0 = fma_f32x2(wy[r], r0, s0);
      s1 = fma_f32x2(wy[r], r1, s1);
    }
    fetch(j + ACC_ST - 1);
    __pipeline_wait_prior(ACC_ST - 1);
    float b0r, b0i, b1r, b1i;
    f32x2_split(s0, b0r, b0i);
    f32x2_split(s1, b1r, b1i);
    const float4* slot = pk + (j % ACC_ST) * 2 * ACC_T + tid;
    const float4 ra = slot[0], rb = slot[ACC_T];  // rb: stale for the odd filter's copy, unused then
    float im0, re0, im1, re1, d0, d1;
    acc_cross(ra, b0r, b0i, im0, re0);
    acc_cross(rb, b1r, b1i, im1, re1);
    atan2_phase_pair(im0, re0, im1, re1, d0, d1);
    acc_add(a, ra, b0r, b0i, d0, u, v);
    if (2 * j + 1 < F) acc_add(a, rb, b1r, b1i, d1, u, v);
  }
  __pipeline_wait_prior(0);
#pragma unroll
  for (int i = 0; i < 7; i++) sums[i * N + p] = a[i];
}

// the accumulate as a gather from the response planes: the form for planes without tensor maps, and the reference
// the TMA-staged kernel (accumulate_tma.cu) is checked against
void launch_accumulate_gather(const float4* ref4, const float2* R, int F, int ph, int pw, const double* ux,
                              const double* uy, const double* sx, const double* sy, const double2* cs, int W, int H,
                              double* sums, cudaStream_t st) {
  dim3 g(div_up(W, ACC_BX), div_up(H, ACC_BY));
  const size_t sm = (size_t)2 * ACC_ST * ACC_T * sizeof(float4);
  if (F > ACC_MAXF)
    throw Error(OFC_ERR_WINDOW, "too many Gabor filters (" + std::to_string(F) + ") for the CUDA engine");
  raise_smem_limit((const void*)k_accumulate, sm);
  OFC_LAUNCH_PDL(k_accumulate, g, dim3(ACC_BX, ACC_BY), sm, st, ref4, (const float4*)R, F, ph, pw, ux, uy, sx, sy, cs, W, H, sums);
}

// ---------------------------------------------------------------- window moments + solve
// The moments a shape function of order 1 or 2 needs (phaseflow.py:123-161), resolved at compile time:
// sources 0..6 = gxx gxy gyy gxc gyc gcc gw; a moment is (source, px, py); the y pass makes (source, py).
struct MomTable {
  int n = 0, ny = 0, nm = 0;
  int ysrc[32] = {}, ypow[32] = {};
  int mjob[64] = {}, mpx[64] = {};
  int Midx[144] = {}, bidx[12] = {};
  int gcc = 0, gw = 0;
};

__host__ __device__ constexpr MomTable build_table(int order) {
  MomTable T{};
  int uc[12] = {}, ux_[12] = {}, uy_[12] = {};
  int pw1[6][2] = {{0, 0}, {1, 0}, {0, 1}, {2, 0}, {1, 1}, {0, 2}};
  int npw = order == 1 ? 3 : 6;
  int n = 0;
  uc[n] = 0; ux_[n] = 0; uy_[n] = 0; n++;
  uc[n] = 1; ux_[n] = 0; uy_[n] = 0; n++;
  for (int i = 1; i < npw; i++)
    for (int c = 0; c < 2; c++) { uc[n] = c; ux_[n] = pw1[i][0]; uy_[n] = pw1[i][1]; n++; }
  T.n = n;
  // moment list
  int msrc[64] = {}, mx[64] = {}, my[64] = {};
  int nm = 0;
  auto find_or_add = [&](int s, int px, int py) {
    for (int i = 0; i < nm; i++)
      if (msrc[i] == s && mx[i] == px && my[i] == py) return i;
    msrc[nm] = s; mx[nm] = px; my[nm] = py;
    return nm++;
  };
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      int a = uc[i] < uc[j] ? uc[i] : uc[j], b = uc[i] < uc[j] ? uc[j] : uc[i];
      int key = a == 0 ? (b == 0 ? 0 : 1) : 2;
      T.Midx[i * n + j] = find_or_add(key, ux_[i] + ux_[j], uy_[i] + uy_[j]);
    }
  for (int i = 0; i < n; i++) T.bidx[i] = find_or_add(3 + uc[i], ux_[i], uy_[i]);
  T.gcc = find_or_add(5, 0, 0);
  T.gw = find_or_add(6, 0, 0);
  T.nm = nm;
  int ny = 0;
  for (int m = 0; m < nm; m++) {
    int j = -1;
    for (int q = 0; q < ny; q++)
      if (T.ysrc[q] == msrc[m] && T.ypow[q] == my[m]) j = q;
    if (j < 0) { T.ysrc[ny] = msrc[m]; T.ypow[ny] = my[m]; j = ny++; }
    T.mjob[m] = j;
    T.mpx[m] = mx[m];
  }
  T.ny = ny;
  return T;
}

int moment_yplanes(int order) { return build_table(order).ny; }

// The window taps k(t) t^p are symmetric in t for even p and antisymmetric for odd p, so each pass pairs
// the samples at +t and -t: sum_t k(t) t^p a(q + t) = [p == 0] k(0) a(q) + sum_{t >= 1} k(t) t^p (a(q + t) +- a(q - t)),
// which halves the float64 multiply-adds (the passes are float64-throughput bound).
template <int ORDER>
__global__ void __launch_bounds__(128) k_moments_y(const double* __restrict__ sums, int W, int H,
                                                   const double* __restrict__ mtaps, int r,
                                                   double* __restrict__ yplanes) {
  constexpr MomTable T = build_table(ORDER);
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  const size_t N = (size_t)W * H;
  const int K = 2 * r + 1;
  double acc[T.ny];
#pragma unroll
  for (int j = 0; j < T.ny; j++) acc[j] = 0;
#pragma unroll
  for (int j = 0; j < T.ny; j++)
    acc[j] = T.ypow[j] == 0 ? mtaps[r] * sums[(size_t)T.ysrc[j] * N + (size_t)y * W + x] : 0.0;
  for (int t = 1; t <= r; t++) {
    const size_t op = (size_t)min(y + t, H - 1) * W + x, om = (size_t)max(y - t, 0) * W + x;
#pragma unroll
    for (int src = 0; src < 7; src++) {
      bool used = false;
#pragma unroll
      for (int j = 0; j < T.ny; j++) used |= T.ysrc[j] == src;
      if (!used) continue;
      const double ap = sums[(size_t)src * N + op], am = sums[(size_t)src * N + om];
      const double sp = ap + am, dm = ap - am;
#pragma unroll
      for (int j = 0; j < T.ny; j++)
        if (T.ysrc[j] == src) acc[j] = fma(mtaps[T.ypow[j] * K + r + t], (T.ypow[j] & 1) ? dm : sp, acc[j]);
    }
  }
  size_t p = (size_t)y * W + x;
#pragma unroll
  for (int j = 0; j < T.ny; j++) yplanes[j * N + p] = acc[j];
}

// Every inner loop below runs over a constant trip count with a guard (k < j rather than a bound of j): a bound
// that depends on the outer index can leave the inner loop rolled, and the matrix then lives in local memory.
// One division per pivot: the factor's column and both substitutions multiply by the pivot's reciprocal.
template <int N>
__device__ __forceinline__ bool cholesky_solve_dev(double (&M)[N * N], double (&b)[N]) {
  bool okp = true;
  double il[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    double d = M[j * N + j];
#pragma unroll
    for (int k = 0; k < N; k++)
      if (k < j) d -= M[j * N + k] * M[j * N + k];
    okp &= d > 0.0 && d <= DBL_MAX;  // a failed pivot goes on with meaningless values and reports false
    // the substitutions below read the pivots only as 1 / l: one reciprocal square root instead of a square root and
    // a division (each a sequence of dependent float64 instructions)
    il[j] = rsqrt(d);
#pragma unroll
    for (int i = 0; i < N; i++) {
      if (i <= j) continue;
      double s = M[i * N + j];
#pragma unroll
      for (int k = 0; k < N; k++)
        if (k < j) s -= M[i * N + k] * M[j * N + k];
      M[i * N + j] = s * il[j];
    }
  }
#pragma unroll
  for (int i = 0; i < N; i++) {
    double s = b[i];
#pragma unroll
    for (int k = 0; k < N; k++)
      if (k < i) s -= M[i * N + k] * b[k];
    b[i] = s * il[i];
  }
#pragma unroll
  for (int i = N - 1; i >= 0; i--) {
    double s = b[i];
#pragma unroll
    for (int k = 0; k < N; k++)
      if (k > i) s -= M[k * N + i] * b[k];
    b[i] = s * il[i];
  }
  bool fin = okp;
#pragma unroll
  for (int i = 0; i < N; i++) fin &= isfinite(b[i]);
  return fin;
}

template <int ORDER>
__global__ void __launch_bounds__(128) k_moments_x_solve(const double* __restrict__ yplanes,
                                                         const double* __restrict__ uxin,
                                                         const double* __restrict__ uyin, int W, int H,
                                                         const double* __restrict__ mtaps, int r,
                                                         double* __restrict__ oux, double* __restrict__ ouy,
                                                         double* __restrict__ energy, double* __restrict__ resid,
                                                         double* __restrict__ slope) {
  constexpr MomTable T = build_table(ORDER);
  constexpr int n = ORDER == 1 ? 6 : 12;
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  const size_t N = (size_t)W * H;
  const int K = 2 * r + 1;
  // one pass over the tap pairs t = 1..r with every moment's accumulator live (independent chains)
  double m[T.nm];
  const double* row = yplanes + (size_t)y * W;
#pragma unroll
  for (int i = 0; i < T.nm; i++) m[i] = T.mpx[i] == 0 ? mtaps[r] * row[(size_t)T.mjob[i] * N + x] : 0.0;
  for (int t = 1; t <= r; t++) {
    const int xp = min(x + t, W - 1), xm = max(x - t, 0);
#pragma unroll
    for (int j = 0; j < T.ny; j++) {
      const double ap = row[(size_t)j * N + xp], am = row[(size_t)j * N + xm];
      const double sp = ap + am, dm = ap - am;
#pragma unroll
      for (int i = 0; i < T.nm; i++)
        if (T.mjob[i] == j) m[i] = fma(mtaps[T.mpx[i] * K + r + t], (T.mpx[i] & 1) ? dm : sp, m[i]);
    }
  }
  const size_t p = (size_t)y * W + x;
  double M[n * n], b[n], b0[n];
#pragma unroll
  for (int i = 0; i < n * n; i++) M[i] = m[T.Midx[i]];
#pragma unroll
  for (int i = 0; i < n; i++) b0[i] = b[i] = m[T.bidx[i]];
  const double m00 = M[0], m11 = M[n + 1], m01 = M[1];
  const double e = m00 + m11;
  const double det2 = m00 * m11 - m01 * m01;
  energy[p] = e;
  bool ok = det2 > APERTURE_TOL * e * e;
  if (ok) {
    double tr = 0;
#pragma unroll
    for (int i = 0; i < n; i++) tr += M[i * n + i];
    double ridge = (1e-12 / n) * tr;
#pragma unroll
    for (int i = 0; i < n; i++) M[i * n + i] += ridge;
    ok = cholesky_solve_dev<n>(M, b);
  }
  if (ok) {
    double fit = 0;
#pragma unroll
    for (int i = 0; i < n; i++) fit += b[i] * b0[i];
    double rr = m[T.gcc] - fit;
    resid[p] = sqrt(fmax(rr, 0.0) / (m[T.gw] + 1e-30));
    oux[p] = b[0];
    ouy[p] = b[1];
#pragma unroll
    for (int i = 0; i < 4; i++) slope[i * N + p] = b[2 + i];
  } else {
    resid[p] = PI;
    oux[p] = uxin[p];
    ouy[p] = uyin[p];
#pragma unroll
    for (int i = 0; i < 4; i++) slope[i * N + p] = 0.0;
  }
}

// ---- window moments for the default window (r = MOM_R = 16, 33 taps) through shared memory
// Both passes walk the tap pairs outward from a thread's RB consecutive outputs with two sliding register windows
// (the RB samples at +t and the RB at -t; a step of t shifts each by one and loads one sample), so RB outputs take
// RB + 32 shared-memory loads and 2 RB + RB x powers live values.
// outputs j of powers 0 .. NP - 1 from the samples v(i), i = 0 .. RB + 31 (output j's centre at i = j + 16)
template <int RB, int NP, class V>
__device__ __forceinline__ void mom_slide(V v, const MomTaps& tp, double (&acc)[RB][NP]) {
  constexpr int R = MOM_R;
  double up[RB], dn[RB];
#pragma unroll
  for (int j = 0; j < RB; j++) {
#pragma unroll
    for (int p = 0; p < NP; p++) acc[j][p] = p == 0 ? tp.k[0][0] * v(j + R) : 0.0;
    up[j] = v(j + R + 1);
    dn[j] = v(j + R - 1);
  }
#pragma unroll
  for (int t = 1; t <= R; t++) {
#pragma unroll
    for (int j = 0; j < RB; j++) {
      const double sp = up[j] + dn[j], dm = up[j] - dn[j];
#pragma unroll
      for (int p = 0; p < NP; p++) acc[j][p] = fma(tp.k[p][t], (p & 1) ? dm : sp, acc[j][p]);
    }
    if (t < R) {
#pragma unroll
      for (int j = 0; j + 1 < RB; j++) up[j] = up[j + 1];
      up[RB - 1] = v(R + t + RB);
#pragma unroll
      for (int j = RB - 1; j > 0; j--) dn[j] = dn[j - 1];
      dn[0] = v(R - t - 1);
    }
  }
}

// the y-planes of a source: the number of y powers it feeds (a prefix 0 .. np - 1) and the plane of each
struct SrcPlanes {
  int np[7] = {};
  int plane[7][5] = {};
};
__host__ __device__ constexpr SrcPlanes build_src_planes(int order) {
  SrcPlanes r{};
  const MomTable T = build_table(order);
  for (int q = 0; q < T.ny; q++) {
    r.plane[T.ysrc[q]][T.ypow[q]] = q;
    if (T.ypow[q] + 1 > r.np[T.ysrc[q]]) r.np[T.ysrc[q]] = T.ypow[q] + 1;
  }
  return r;
}
__constant__ SrcPlanes c_src_planes[2] = {build_src_planes(1), build_src_planes(2)};

// y pass: a block takes 32 columns x 8 RY rows of one source plane (blockIdx.z) and its 2r halo rows into shared memory
// (asynchronous copies), a warp RY rows of them. Bound by the float64 pipe (63 % busy) and its 15 output planes; the loads
// of a tile wait behind other blocks' arithmetic. Order 1 at 2048^2: 0.162 ms with 6 rows per warp lane and 3 blocks of 256
// threads per SM (78 registers) against 0.208 ms for 36 global loads per 4 outputs; 4 rows 0.169, 8 rows (128 registers)
// 0.189. Order 2 (up to 5 powers) keeps 4 rows: 64 registers without spills.
constexpr int MY_W = 8;
template <int ORDER>
struct MomY {
  static constexpr int RY = ORDER == 1 ? 6 : 4, MINB = ORDER == 1 ? 3 : 4;
};
template <int ORDER>
__global__ void __launch_bounds__(32 * MY_W, MomY<ORDER>::MINB) k_moments_y_rb(const double* __restrict__ sums, int W, int H, MomTaps tp,
                                                             double* __restrict__ yplanes) {
  grid_dep_wait();
  constexpr int R = MOM_R, RY = MomY<ORDER>::RY, TB = MY_W * RY, NR = TB + 2 * R;
  static_assert(NR % MY_W == 0, "whole rows of the tile per warp");
  __shared__ double tile[NR * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, src = blockIdx.z;
  const int x = blockIdx.x * 32 + lane, y0 = blockIdx.y * TB;
  const size_t N = (size_t)W * H;
  const double* plane = sums + (size_t)src * N + x;
  if (x < W) {
#pragma unroll
    for (int i = 0; i < NR / MY_W; i++) {
      const int r = wid + MY_W * i;
      __pipeline_memcpy_async(tile + r * 32 + lane, plane + (size_t)min(max(y0 - R + r, 0), H - 1) * W, sizeof(double));
    }
  }
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
  const int yb = y0 + wid * RY;
  if (x >= W || yb >= H) return;
  const double* t0 = tile + wid * RY * 32 + lane;
  const SrcPlanes& SP = c_src_planes[ORDER - 1];
  auto run = [&](auto npc) {
    constexpr int NP = decltype(npc)::value;
    double acc[RY][NP];
    mom_slide<RY, NP>([&](int i) { return t0[i * 32]; }, tp, acc);
#pragma unroll
    for (int p = 0; p < NP; p++) {
      double* o = yplanes + (size_t)SP.plane[src][p] * N + (size_t)yb * W + x;
#pragma unroll
      for (int j = 0; j < RY; j++) {
        if (yb + j < H) o[(size_t)j * W] = acc[j][p];
      }
    }
  };
  const int np = SP.np[src];  // order 1: 3 (products), 2 (right sides), 1; order 2: 5, 3, 1
  if (np == 1) run(std::integral_constant<int, 1>{});
  else if (np == 3) run(std::integral_constant<int, 3>{});
  else if (ORDER == 1) run(std::integral_constant<int, 2>{});
  else run(std::integral_constant<int, 5>{});
}

// x pass + solve: a block owns a row segment of SEG = 32 RX pixels and has G warps that share out its y-planes (a fixed
// balanced schedule). A warp stages its plane's segment and 2r halo in a buffer of its own (double-buffered asynchronous
// copies; only warp barriers), a lane forms the moments of RX consecutive pixels (an odd RX keeps the lanes' reads on
// distinct banks) and writes them into a shared tile of nm x SEG. Then the block's threads solve a pixel each from the
// tile. The float64 pipe bounds it (69 % busy; the solve is a third of its work), and a lane's sample loads next:
// (RX + 32) / RX per pixel and plane. Order 1 at 2048^2: 0.334 ms with 5 pixels per lane, 4 warps, 4 blocks per SM (117
// registers) against 0.393 ms for two groups of 64 threads with 3 pixels each; 3 pixels 0.36-0.38, 7 pixels 0.395, 5
// warps at 96 registers 0.335. Order 2 (59 moments per pixel bound the tile, the 12 x 12 solve the registers) at 512^2:
// 88 us with 3 pixels per lane against 131 us with one.
template <int ORDER>
struct MomX {
  static constexpr int RX = ORDER == 1 ? 5 : 3, G = 4, MINB = ORDER == 1 ? 4 : 2;
  static constexpr int NT = 32 * G, SEG = 32 * RX, WIN = SEG + 2 * MOM_R;
  static constexpr size_t smem() { return (size_t)(2 * G * WIN + build_table(ORDER).nm * SEG) * sizeof(double); }
};

// Per y-plane of an order: the number of x powers it feeds (always a prefix 0 .. npow - 1 of the powers) and the
// moment-tile row of each, so that one plane body per power count serves every plane
struct PlaneRows {
  int npow[32] = {};
  int mi[32][5] = {};
};
__host__ __device__ constexpr PlaneRows build_plane_rows(int order) {
  PlaneRows r{};
  const MomTable T = build_table(order);
  for (int q = 0; q < T.ny; q++) {
    for (int p = 0; p < 5; p++) r.mi[q][p] = -1;
    int np = 0;
    for (int m = 0; m < T.nm; m++)
      if (T.mjob[m] == q) {
        r.mi[q][T.mpx[m]] = m;
        if (T.mpx[m] + 1 > np) np = T.mpx[m] + 1;
      }
    r.npow[q] = np;
  }
  return r;
}
__host__ __device__ constexpr bool plane_rows_are_prefixes(int order) {
  const PlaneRows r = build_plane_rows(order);
  const MomTable T = build_table(order);
  for (int q = 0; q < T.ny; q++)
    for (int p = 0; p < r.npow[q]; p++)
      if (r.mi[q][p] < 0) return false;
  return true;
}
static_assert(plane_rows_are_prefixes(1) && plane_rows_are_prefixes(2), "a y-plane feeds a gap in the powers");
__host__ __device__ constexpr int max_plane_powers(int order) {
  const PlaneRows r = build_plane_rows(order);
  int mx = 0;
  for (int q = 0; q < build_table(order).ny; q++) mx = r.npow[q] > mx ? r.npow[q] : mx;
  return mx;
}
static_assert(max_plane_powers(1) == 3 && max_plane_powers(2) == 5, "the bodies' power counts");
__constant__ PlaneRows c_plane_rows[2] = {build_plane_rows(1), build_plane_rows(2)};

// the warps' y-planes: the most costly plane (2 + powers operations per tap pair) first, each to the least loaded warp
template <int G>
struct PlaneShare {
  int n[G] = {};
  int q[G][32] = {};
};
template <int G>
__host__ __device__ constexpr PlaneShare<G> build_share(int order) {
  PlaneShare<G> s{};
  const PlaneRows r = build_plane_rows(order);
  const int ny = build_table(order).ny;
  int load[G] = {};
  for (int np = 5; np >= 1; np--)
    for (int q = 0; q < ny; q++) {
      if (r.npow[q] != np) continue;
      int g = 0;
      for (int k = 1; k < G; k++)
        if (load[k] < load[g]) g = k;
      s.q[g][s.n[g]++] = q;
      load[g] += np == 1 ? 2 : 2 + np;
    }
  return s;
}
__constant__ PlaneShare<MomX<1>::G> c_share1 = build_share<MomX<1>::G>(1);
__constant__ PlaneShare<MomX<2>::G> c_share2 = build_share<MomX<2>::G>(2);

template <int ORDER>
__global__ void __launch_bounds__(MomX<ORDER>::NT, MomX<ORDER>::MINB) k_moments_x_solve_rb(const double* __restrict__ yplanes,
                                                               const double* __restrict__ uxin,
                                                               const double* __restrict__ uyin, int W, int H,
                                                               MomTaps tp, double* __restrict__ oux,
                                                               double* __restrict__ ouy, double* __restrict__ energy,
                                                               double* __restrict__ resid, double* __restrict__ slope) {
  grid_dep_wait();
  constexpr MomTable T = build_table(ORDER);
  constexpr int n = ORDER == 1 ? 6 : 12;
  constexpr int RX = MomX<ORDER>::RX, G = MomX<ORDER>::G, NT = MomX<ORDER>::NT, SEG = MomX<ORDER>::SEG;
  constexpr int WIN = MomX<ORDER>::WIN, NI = WIN / 32;
  extern __shared__ double smd[];
  double* mom = smd + 2 * G * WIN;
  const int tid = threadIdx.x, g = tid >> 5, lane = tid & 31, y = blockIdx.y, x0 = blockIdx.x * SEG;
  const size_t N = (size_t)W * H;
  const auto& SH = [] () -> const auto& { if constexpr (ORDER == 1) return c_share1; else return c_share2; }();
  const PlaneRows& PR = c_plane_rows[ORDER - 1];
  double* gb = smd + 2 * WIN * g;  // the warp's two buffers
  int off[NI];                     // the lane's samples of a row segment, edges replicated
#pragma unroll
  for (int i = 0; i < NI; i++) off[i] = min(max(x0 - MOM_R + lane + 32 * i, 0), W - 1);
  const int cnt = SH.n[g];
  auto fetch = [&](int k) {
    if (k < cnt) {
      const double* row = yplanes + (size_t)SH.q[g][k] * N + (size_t)y * W;
      double* dst = gb + (k & 1) * WIN + lane;
#pragma unroll
      for (int i = 0; i < NI; i++) __pipeline_memcpy_async(dst + 32 * i, row + off[i], sizeof(double));
    }
    __pipeline_commit();
  };
  fetch(0);
#pragma unroll 1
  for (int k = 0; k < cnt; k++) {
    fetch(k + 1);
    __pipeline_wait_prior(1);
    __syncwarp();
    const int q = SH.q[g][k];
    const double* wb = gb + (k & 1) * WIN + lane * RX;
    auto run = [&](auto npc) {
      constexpr int NP = decltype(npc)::value;
      double acc[RX][NP];
      mom_slide<RX, NP>([&](int i) { return wb[i]; }, tp, acc);
#pragma unroll
      for (int p = 0; p < NP; p++) {
        double* o = mom + PR.mi[q][p] * SEG + lane * RX;
#pragma unroll
        for (int j = 0; j < RX; j++) o[j] = acc[j][p];
      }
    };
    const int np = PR.npow[q];  // order 1: at most 3 (powers 0 .. 2); order 2: at most 5
    if (np == 1) run(std::integral_constant<int, 1>{});
    else if (np == 2) run(std::integral_constant<int, 2>{});
    else if (ORDER == 1 || np == 3) run(std::integral_constant<int, 3>{});
    else if constexpr (ORDER > 1) {
      if (np == 4) run(std::integral_constant<int, 4>{});
      else run(std::integral_constant<int, 5>{});
    }
    __syncwarp();  // the buffer of plane k is free for plane k + 2
  }
  __pipeline_wait_prior(0);
  __syncthreads();
#pragma unroll 1
  for (int s = tid; s < SEG; s += NT) {
    const int x = x0 + s;
    if (x >= W) continue;
    double m[T.nm];
#pragma unroll
    for (int k = 0; k < T.nm; k++) m[k] = mom[k * SEG + s];
    const size_t p = (size_t)y * W + x;
    double M[n * n], b[n], b0[n];
#pragma unroll
    for (int k = 0; k < n * n; k++) M[k] = m[T.Midx[k]];
#pragma unroll
    for (int k = 0; k < n; k++) b0[k] = b[k] = m[T.bidx[k]];
    const double m00 = M[0], m11 = M[n + 1], m01 = M[1];
    const double e = m00 + m11;
    const double det2 = m00 * m11 - m01 * m01;
    energy[p] = e;
    bool ok = det2 > APERTURE_TOL * e * e;
    if (ok) {
      double tr = 0;
#pragma unroll
      for (int k = 0; k < n; k++) tr += M[k * n + k];
      double ridge = (1e-12 / n) * tr;
#pragma unroll
      for (int k = 0; k < n; k++) M[k * n + k] += ridge;
      ok = cholesky_solve_dev<n>(M, b);
    }
    if (ok) {
      double fit = 0;
#pragma unroll
      for (int k = 0; k < n; k++) fit += b[k] * b0[k];
      double rr = m[T.gcc] - fit;
      resid[p] = sqrt(fmax(rr, 0.0) / (m[T.gw] + 1e-30));
      oux[p] = b[0];
      ouy[p] = b[1];
#pragma unroll
      for (int k = 0; k < 4; k++) slope[k * N + p] = b[2 + k];
    } else {
      resid[p] = PI;
      oux[p] = uxin[p];
      ouy[p] = uyin[p];
#pragma unroll
      for (int k = 0; k < 4; k++) slope[k * N + p] = 0.0;
    }
  }
}

template <int ORDER>
static void launch_moments_rb(const double* sums, const double* ux, const double* uy, int W, int H, const MomTaps& tp,
                              double* yplanes, double* oux, double* ouy, double* energy, double* resid, double* slope,
                              cudaStream_t st) {
  dim3 gy(div_up(W, 32), div_up(H, MY_W * MomY<ORDER>::RY), 7);
  OFC_LAUNCH_PDL(k_moments_y_rb<ORDER>, gy, 32 * MY_W, 0, st, sums, W, H, tp, yplanes);
  const size_t sm = MomX<ORDER>::smem();
  raise_smem_limit((const void*)k_moments_x_solve_rb<ORDER>, sm);
  dim3 gx(div_up(W, MomX<ORDER>::SEG), H);
  OFC_LAUNCH_PDL(k_moments_x_solve_rb<ORDER>, gx, MomX<ORDER>::NT, sm, st, yplanes, ux, uy, W, H, tp, oux, ouy, energy, resid,
             slope);
}

void launch_moments_solve(const double* sums, const double* ux, const double* uy, int W, int H, int order,
                          const double* mtaps, int r, const MomTaps& tp, double* yplanes, double* oux, double* ouy,
                          double* energy, double* resid, double* slope, cudaStream_t st) {
  if (r == MOM_R) {
    if (order == 1) launch_moments_rb<1>(sums, ux, uy, W, H, tp, yplanes, oux, ouy, energy, resid, slope, st);
    else launch_moments_rb<2>(sums, ux, uy, W, H, tp, yplanes, oux, ouy, energy, resid, slope, st);
    return;
  }
  dim3 g(div_up(W, 128), H);
  if (order == 1) {
    OFC_LAUNCH(k_moments_y<1>, g, 128, 0, st, sums, W, H, mtaps, r, yplanes);
    OFC_LAUNCH(k_moments_x_solve<1>, g, 128, 0, st, yplanes, ux, uy, W, H, mtaps, r, oux, ouy, energy, resid, slope);
  } else {
    OFC_LAUNCH(k_moments_y<2>, g, 128, 0, st, sums, W, H, mtaps, r, yplanes);
    OFC_LAUNCH(k_moments_x_solve<2>, g, 128, 0, st, yplanes, ux, uy, W, H, mtaps, r, oux, ouy, energy, resid, slope);
  }
}

// ---------------------------------------------------------------- energy median and reset
// The median of the energy (np.median, phaseflow.py:149-151) by an exact select over order-preserving keys, and the reset
// that reads it:
// 1. the range of the energies and the reset rule (phaseflow.rs:846-854): when every energy is above 1e-9 max + 1e-30 no
//    pixel is reset, and unless the caller needs the median nothing more is done;
// 2. a histogram of 4096 equal parts of the keys' range, and the part that holds the element of rank n / 2;
// 3. that part's elements as a candidate list, the largest key below it, and the select among the candidates (their range
//    split again while there are more than MED_LIST, then by counting);
// 4. the reset of each pixel below the threshold.
// Blocks wait for each other only at the hardware's cluster barrier: no wait can give up, a median shares the SMs with
// other streams' kernels, and the launches take programmatic dependencies like their neighbours. One cooperative launch of
// 1024-thread blocks with grid barriers, as it was before, is no faster (us per pair before -> now: 128^2 1290 -> 1212, 256^2
// 1637 -> 1612, 512^2 of order 2 4220 -> 4192, 1024^2 8690 -> 8610, 2048^2 30930 -> 30850).
// Small images are bound by the launches' latency: up to MED_CLUSTER_N energies one cluster of 8 blocks does it all
// (k_median_cluster; 300 x 300 pairs 2228 us against 2252 with a launch per step, 360 x 360 3623 against 3593). Beyond, a
// launch per step over the whole chip, whose last block to finish picks (k_median_range, k_median_hist, k_median_select,
// k_median_reset). us per launch of a forced median at 2048^2: range 14, histogram 15 to 19, select 21. Where the energies'
// range is stretched the part is wide, the candidates many, and the last block alone goes through them: select 97 with ties
// of three values, 395 with one zero energy among ordinary ones; a frame whose dark 60 % span five octaves 21. A pair of
// 2048^2 pixels, 60 % of them dark, takes 45.7 ms with it as it did with the cooperative form.
constexpr size_t MED_CLUSTER_N = 98304;
__device__ __forceinline__ unsigned long long okey(double v) {  // order-preserving key of a double
  unsigned long long u = (unsigned long long)__double_as_longlong(v);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ULL);
}
__device__ __forceinline__ double okey_inv(unsigned long long k) {
  unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k;
  return __longlong_as_double((long long)u);
}

constexpr int MED_LIST = 256;  // candidates that are selected by counting (the square of their number)

__device__ __forceinline__ EnergyStats::Half median_start() {
  EnergyStats::Half h{};
  h.lo = h.first = ~0ull;
  return h;
}
__global__ void k_stats_init(EnergyStats* s) {
  s->median = 0.0;
  for (int i = 0; i < 2; i++) s->half[i] = median_start();
}

// every energy is above 1e-9 max + 1e-30 (lo, hi: the smallest and largest key, ~0 and 0 where all are NaN)
__device__ __forceinline__ bool median_skips(unsigned long long lo, unsigned long long hi, bool nan) {
  const double vlo = okey_inv(lo), vhi = okey_inv(hi);
  return !nan && vhi <= DBL_MAX / 2 && vlo > 1e-9 * vhi + 1e-30;
}
// log2 of the keys per part where [lo, hi] is split into at most 2^log_bins parts
__device__ __forceinline__ int median_shift(unsigned long long lo, unsigned long long hi, int log_bins) {
  return max(64 - __clzll((long long)(hi - lo)) - log_bins, 0);
}
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}

// f(energy, index) for the thread's energies, the pairs i0, i0 + step, ... of n: the first E pairs, which the caller loaded
// into v, from registers, later ones from memory, four loads at a time. e: 16-byte aligned
template <class I>
__device__ __forceinline__ double2 load_pair(const double* __restrict__ e, I n, I i) {
  if (2 * i + 1 < n) return *reinterpret_cast<const double2*>(e + 2 * i);
  return make_double2(2 * i < n ? e[2 * i] : 0.0, 0.0);
}
template <int E, class I>
__device__ __forceinline__ void load_energies(const double* __restrict__ e, I n, I i0, I step, double2 (&v)[E]) {
#pragma unroll
  for (int u = 0; u < E; u++) v[u] = load_pair(e, n, i0 + u * step);
}
template <int E, class I, class F>
__device__ __forceinline__ void each_energy(const double* __restrict__ e, I n, I i0, I step, const double2 (&v)[E], F f) {
  auto both = [&](double2 w, I i) {
    if (2 * i < n) f(w.x, 2 * i);
    if (2 * i + 1 < n) f(w.y, 2 * i + 1);
  };
#pragma unroll
  for (int u = 0; u < E; u++) both(v[u], i0 + u * step);
  for (I i = i0 + E * step; 2 * i < n; i += 4 * step) {
    double2 w[4];
    load_energies(e, n, i, step, w);
#pragma unroll
    for (int u = 0; u < 4; u++) both(w[u], i + u * step);
  }
}

// the smallest and largest key of a block's energies and whether one is NaN, into shared memory (~0, 0 and 0 before). The
// caller synchronises
template <int E, class I>
__device__ __forceinline__ void energy_range(const double* __restrict__ e, I n, I i0, I step, const double2 (&v)[E],
                                             unsigned long long* slo, unsigned long long* shi, unsigned* snan) {
  unsigned long long lo = ~0ull, hi = 0;
  bool nan = false;
  each_energy(e, n, i0, step, v, [&](double x, auto) {
    if (x != x) {
      nan = true;
    } else {
      const unsigned long long k = okey(x);
      lo = k < lo ? k : lo;
      hi = k > hi ? k : hi;
    }
  });
  __syncwarp();
  lo = ~warp_max64(~lo);
  hi = warp_max64(hi);
  nan = __any_sync(0xffffffffu, nan);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(slo, lo);
    atomicMax(shi, hi);
    if (nan) atomicOr(snan, 1u);
  }
}

// inclusive sums of v over the threads of a block of T; tot: T / 32 values of shared memory, the last of which holds the
// sum over the block afterwards. The caller synchronises before tot is used again
template <int T>
__device__ long long block_scan(long long v, long long* tot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long w = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += w;
  }
  if (lane == 31) tot[wid] = v;
  __syncthreads();
  if (wid == 0) {
    long long w = lane < T / 32 ? tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    if (lane < T / 32) tot[lane] = w;
  }
  __syncthreads();
  return v + (wid ? tot[wid - 1] : 0);
}

// the bin of BINS counts (count(i)) that holds `rank`, the number of elements in the bins before it and its own; every
// thread of the block of T gets them. The counts sum to more than rank
template <int T, int BINS, class Count>
__device__ void block_pick(Count count, long long rank, int& bin, long long& before, unsigned& in) {
  constexpr int PER = BINS / T;
  __shared__ long long tot[T / 32], sh_before;
  __shared__ int sh_bin;
  __shared__ unsigned sh_in;
  unsigned c[PER];
  long long loc = 0;
#pragma unroll
  for (int j = 0; j < PER; j++) {
    c[j] = count((int)threadIdx.x * PER + j);
    loc += c[j];
  }
  long long acc = block_scan<T>(loc, tot) - loc;
  if (acc <= rank && rank < acc + loc) {  // exactly one thread
    bool found = false;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      if (!found && rank < acc + c[j]) {
        found = true;
        sh_bin = (int)threadIdx.x * PER + j;
        sh_before = acc;
        sh_in = c[j];
      }
      if (!found) acc += c[j];
    }
  }
  __syncthreads();
  bin = sh_bin;
  before = sh_before;
  in = sh_in;
  __syncthreads();
}

// the key of rank `rank` among the nc <= MED_LIST keys (shared memory) by counting, and how many of them are less; every
// thread of the block gets both. nc > rank
__device__ void count_select(const unsigned long long* keys, unsigned nc, long long rank, unsigned long long& key,
                             long long& less) {
  __shared__ unsigned long long sh_key;
  __shared__ long long sh_less;
  for (unsigned t = threadIdx.x; t < nc; t += blockDim.x) {
    const unsigned long long k = keys[t];
    unsigned lt = 0, le = 0;
    for (unsigned i = 0; i < nc; i++) {
      lt += keys[i] < k;
      le += keys[i] <= k;
    }
    if ((long long)lt <= rank && rank < (long long)le) {  // the equal keys of that rank write the same values
      sh_key = k;
      sh_less = lt;
    }
  }
  __syncthreads();
  key = sh_key;
  less = sh_less;
}

// the largest of the nc keys at(i) below `key`, or `floor` if that is larger; every thread of the block gets it
template <class At>
__device__ unsigned long long block_below(At at, unsigned nc, unsigned long long key, unsigned long long floor) {
  __shared__ unsigned long long sh;
  if (threadIdx.x == 0) sh = floor;
  __syncthreads();
  unsigned long long best = 0;
  for (unsigned i = threadIdx.x; i < nc; i += blockDim.x) {
    const unsigned long long k = at(i);
    if (k < key && k > best) best = k;
  }
  __syncwarp();
  best = warp_max64(best);
  if ((threadIdx.x & 31) == 0 && best) atomicMax(&sh, best);
  __syncthreads();
  return sh;
}

struct ResetPlanes {  // the planes of the reset; ux null: none
  const double *uxin, *uyin;
  double *ux, *uy, *resid, *slope;
};
__device__ __forceinline__ void reset_pixel(const ResetPlanes& r, size_t n, size_t p) {
  r.ux[p] = r.uxin[p];
  r.uy[p] = r.uyin[p];
  r.resid[p] = PI;
  for (int i = 0; i < 4; i++) r.slope[i * n + p] = 0.0;
}

// ---- one cluster: the steps' results in the blocks' shared memory
constexpr int MC_B = 8, MC_T = 512, MC_E = 4;  // blocks, threads, pairs of energies a thread keeps in registers
constexpr int MC_LOG = 12, MC_BINS = 1 << MC_LOG;  // parts of a histogram
static_assert(MC_BINS == MC_B * MC_T, "a bin per thread of the cluster");

__global__ void __cluster_dims__(MC_B, 1, 1) __launch_bounds__(MC_T, 2)
    k_median_cluster(const double* __restrict__ e, unsigned n, EnergyStats* s, int force, ResetPlanes rp) {
  grid_dep_wait();
  namespace cg = cooperative_groups;
  __shared__ unsigned h[MC_BINS];
  __shared__ unsigned long long keys[MED_LIST];
  __shared__ unsigned long long lo, hi, below, all_lo, all_hi, all_below;
  __shared__ unsigned nan, ncand;
  __shared__ bool all_nan;
  __shared__ long long tot[MC_T / 32], sh_before;
  __shared__ int sh_bin;
  __shared__ unsigned sh_in;
  const cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, rank_b = (int)cl.block_rank();
  const unsigned i0 = rank_b * MC_T + tid, step = MC_B * MC_T;
  double2 v[MC_E];
  load_energies(e, n, i0, step, v);
  if (tid == 0) {
    lo = ~0ull;
    hi = below = 0;
    nan = ncand = 0;
  }
  for (int i = tid; i < MC_BINS; i += MC_T) h[i] = 0;
  __syncthreads();
  energy_range(e, n, i0, step, v, &lo, &hi, &nan);
  cl.sync();
  if (tid < 32) {  // a block's range per lane
    const int b = tid % MC_B;
    const unsigned long long l = ~warp_max64(~*cl.map_shared_rank(&lo, b)), m = warp_max64(*cl.map_shared_rank(&hi, b));
    const bool any = __any_sync(0xffffffffu, *cl.map_shared_rank(&nan, b) != 0);
    if (tid == 0) {
      all_lo = l;
      all_hi = m;
      all_nan = any;
    }
  }
  cl.sync();  // the blocks' ranges are read
  const unsigned long long klo = all_lo, khi = all_hi;
  const bool skip = median_skips(klo, khi, all_nan);
  if (!force && skip) return;
  double med = ::nan("");
  if (!all_nan) {
    long long rank = n / 2, less = 0;
    unsigned long long base = klo, width = khi - klo;  // keys of the part: base .. base + width
    for (int shift = median_shift(klo, khi, MC_LOG);; shift = max(shift - MC_LOG, 0)) {
      each_energy(e, n, i0, step, v, [&](double x, auto) {
        const unsigned long long k = okey(x) - base;  // below base: beyond any width
        if (k <= width) atomicAdd(&h[k >> shift], 1u);
      });
      cl.sync();
      // a bin per thread of the cluster: the sums over the blocks, the block's share of the ranks
      unsigned c = 0;
#pragma unroll
      for (int b = 0; b < MC_B; b++) c += cl.map_shared_rank(h, b)[rank_b * MC_T + tid];
      long long excl = block_scan<MC_T>(c, tot) - c;
      cl.sync();
#pragma unroll 1
      for (int b = 0; b < rank_b; b++) excl += cl.map_shared_rank(tot, b)[MC_T / 32 - 1];
      if (excl <= rank && rank < excl + c) {  // exactly one thread of the cluster
#pragma unroll 1
        for (int b = 0; b < MC_B; b++) {
          *cl.map_shared_rank(&sh_bin, b) = rank_b * MC_T + tid;
          *cl.map_shared_rank(&sh_before, b) = excl;
          *cl.map_shared_rank(&sh_in, b) = c;
        }
      }
      for (int i = tid; i < MC_BINS; i += MC_T) h[i] = 0;  // its readers have met
      cl.sync();
      base += (unsigned long long)sh_bin << shift;
      width = (1ull << shift) - 1;
      rank -= sh_before;
      less += sh_before;
      if (shift == 0 || sh_in <= MED_LIST) break;
    }
    // the part's elements into block 0's list (where its keys differ), and the largest key below the part
    const bool list = width > 0;
    unsigned* count = cl.map_shared_rank(&ncand, 0);
    unsigned long long *cand = cl.map_shared_rank(keys, 0), under = 0;
    each_energy(e, n, i0, step, v, [&](double x, auto) {
      const unsigned long long k = okey(x);
      if (k < base) under = k > under ? k : under;
      else if (list && k - base <= width) cand[atomicAdd(count, 1u)] = k;
    });
    __syncwarp();
    under = warp_max64(under);
    if ((tid & 31) == 0 && under) atomicMax(&below, under);
    cl.sync();
    const unsigned nc = *count;
    if (tid < 32) {
      under = warp_max64(*cl.map_shared_rank(&below, tid % MC_B));
      if (tid == 0) all_below = under;
    }
    if (rank_b > 0)
      for (unsigned i = tid; i < nc; i += MC_T) keys[i] = cand[i];
    cl.sync();  // block 0 may end, and every block's own copy is whole
    unsigned long long kmed = base;
    if (list) {
      long long lt;
      count_select(keys, nc, rank, kmed, lt);
      less += lt;
    }
    med = okey_inv(kmed);
    // an even count's lower middle: the same value unless exactly n / 2 elements are below it, then the largest of those
    if (n % 2 == 0 && less >= (long long)(n / 2)) med = (okey_inv(block_below([&](unsigned i) { return keys[i]; }, nc, kmed, all_below)) + med) / 2.0;
  }
  if (i0 == 0) s->median = med;
  if (skip || !rp.ux) return;
  const double thr = 1e-9 * med + 1e-30;
  each_energy(e, n, i0, step, v, [&](double x, unsigned p) {
    if (!(x > thr)) reset_pixel(rp, n, p);
  });
}

// ---- a launch per step
constexpr int ML_T = 512, ML_E = 2;  // threads, pairs of energies a thread keeps in registers
// blocks of a scan: a thread's first ML_E pairs cover n, at most two blocks per SM of 148
static unsigned median_blocks(size_t n) { return std::min(296u, div_up(n, 2 * ML_T * ML_E)); }

// whether this is the last block of the grid to arrive (its writes before are visible to that block); every thread gets it
__device__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) *ticket = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

__global__ void __launch_bounds__(ML_T, 2) k_median_range(const double* __restrict__ e, size_t n, EnergyStats* s, int half) {
  grid_dep_wait();
  const size_t i0 = blockIdx.x * (size_t)ML_T + threadIdx.x, step = (size_t)gridDim.x * ML_T;
  // the other half's start state for the next median (the launches that used it have ended)
  if (i0 == 0) s->half[half ^ 1] = median_start();
  EnergyStats::Half& P = s->half[half];
  __shared__ unsigned long long lo, hi;
  __shared__ unsigned nan;
  double2 v[ML_E];
  load_energies(e, n, i0, step, v);
  if (threadIdx.x == 0) {
    lo = ~0ull;
    hi = 0;
    nan = 0;
  }
  __syncthreads();
  energy_range(e, n, i0, step, v, &lo, &hi, &nan);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMin(&P.lo, lo);
    atomicMax(&P.hi, hi);
    if (nan) atomicOr(&P.nan, 1u);
  }
}

constexpr int ML_LOG = 12, ML_BINS = 1 << ML_LOG;  // parts of a histogram
// the median is not needed
__device__ __forceinline__ bool median_done(const EnergyStats::Half& P, int force) {
  return !force && median_skips(P.lo, P.hi, P.nan != 0);
}

// the last block picks the part and leaves the histogram zero
__global__ void __launch_bounds__(ML_T, 2) k_median_hist(const double* __restrict__ e, size_t n, EnergyStats* s, int half,
                                                       int force, unsigned* hist) {
  grid_dep_wait();
  EnergyStats::Half& P = s->half[half];
  if (P.nan || median_done(P, force)) return;
  __shared__ unsigned h[ML_BINS];
  const unsigned long long base = P.lo;
  const int shift = median_shift(P.lo, P.hi, ML_LOG);
  const size_t i0 = blockIdx.x * (size_t)ML_T + threadIdx.x, step = (size_t)gridDim.x * ML_T;
  double2 v[ML_E];
  load_energies(e, n, i0, step, v);
  for (int i = threadIdx.x; i < ML_BINS; i += ML_T) h[i] = 0;
  __syncthreads();
  each_energy(e, n, i0, step, v, [&](double x, auto) { atomicAdd(&h[(okey(x) - base) >> shift], 1u); });
  __syncthreads();
  for (int i = threadIdx.x; i < ML_BINS; i += ML_T)
    if (h[i]) atomicAdd(&hist[i], h[i]);
  if (!last_block(&P.ticket)) return;
  int bin;
  long long before;
  unsigned in;
  block_pick<ML_T, ML_BINS>([&](int i) { return __ldcg(hist + i); }, (long long)(n / 2), bin, before, in);
  for (int i = threadIdx.x; i < ML_BINS; i += ML_T) hist[i] = 0;
  if (threadIdx.x == 0) {
    P.base = base + ((unsigned long long)bin << shift);
    P.less = before;
    P.shift = shift;
  }
}

// the part's elements as a list, the largest key below the part; the last block selects the median
__global__ void __launch_bounds__(ML_T, 2) k_median_select(const double* __restrict__ e, size_t n, EnergyStats* s, int half,
                                                         int force, unsigned long long* cand) {
  grid_dep_wait();
  EnergyStats::Half& P = s->half[half];
  if (median_done(P, force)) return;
  if (P.nan) {
    if (blockIdx.x == 0 && threadIdx.x == 0) s->median = nan("");
    return;
  }
  __shared__ unsigned h[ML_BINS];
  __shared__ unsigned long long keys[MED_LIST], below, first, last;
  __shared__ unsigned nkeys;
  const unsigned long long base = P.base, width = (1ull << P.shift) - 1;
  const size_t i0 = blockIdx.x * (size_t)ML_T + threadIdx.x, step = (size_t)gridDim.x * ML_T;
  double2 v[ML_E];
  load_energies(e, n, i0, step, v);
  if (threadIdx.x == 0) {
    below = last = 0;
    first = ~0ull;
    nkeys = 0;
  }
  __syncthreads();
  unsigned long long under = 0, lo = ~0ull, hi = 0;
  each_energy(e, n, i0, step, v, [&](double x, auto) {
    const unsigned long long k = okey(x);
    if (k < base) {
      under = k > under ? k : under;
    } else if (k - base <= width) {
      lo = k < lo ? k : lo;
      hi = k > hi ? k : hi;
      cand[atomicAdd(&P.ncand, 1u)] = k;  // the active lanes' additions are made as one
    }
  });
  __syncwarp();
  under = warp_max64(under);
  lo = ~warp_max64(~lo);
  hi = warp_max64(hi);
  if ((threadIdx.x & 31) == 0) {
    if (under) atomicMax(&below, under);
    if (hi) {
      atomicMin(&first, lo);
      atomicMax(&last, hi);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (below) atomicMax(&P.below, below);
    if (last) {
      atomicMin(&P.first, first);
      atomicMax(&P.last, last);
    }
  }
  if (!last_block(&P.ticket)) return;
  const unsigned nc = __ldcg(&P.ncand);
  // f(key) for the candidates from lo to hi
  auto among = [&](auto f) {
    for (unsigned i = threadIdx.x; i < nc; i += 8 * ML_T) {
      unsigned long long k[8];
#pragma unroll
      for (int u = 0; u < 8; u++) k[u] = i + u * ML_T < nc ? __ldcg(cand + i + u * ML_T) : ~0ull;
#pragma unroll
      for (int u = 0; u < 8; u++)
        if (k[u] - lo <= hi - lo) f(k[u]);
    }
  };
  lo = __ldcg(&P.first);
  hi = __ldcg(&P.last);
  long long less = P.less, rank = (long long)(n / 2) - less;
  for (unsigned in = nc; in > MED_LIST && lo != hi;) {  // the candidates' range split again
    const int shift = median_shift(lo, hi, ML_LOG);
    for (int i = threadIdx.x; i < ML_BINS; i += ML_T) h[i] = 0;
    __syncthreads();
    among([&](unsigned long long k) { atomicAdd(&h[(k - lo) >> shift], 1u); });
    __syncthreads();
    int bin;
    long long before;
    block_pick<ML_T, ML_BINS>([&](int i) { return h[i]; }, rank, bin, before, in);
    rank -= before;
    less += before;
    lo += (unsigned long long)bin << shift;
    hi = min(hi, lo + ((1ull << shift) - 1));
  }
  unsigned long long kmed = lo;
  if (lo != hi) {
    among([&](unsigned long long k) { keys[atomicAdd(&nkeys, 1u)] = k; });
    __syncthreads();
    long long lt;
    count_select(keys, nkeys, rank, kmed, lt);
    less += lt;
  }
  double med = okey_inv(kmed);
  // an even count's lower middle: the same value unless exactly n / 2 elements are below it, then the largest of those
  if (n % 2 == 0 && less >= (long long)(n / 2))
    med = (okey_inv(block_below([&](unsigned i) { return __ldcg(cand + i); }, nc, kmed, __ldcg(&P.below))) + med) / 2.0;
  if (threadIdx.x == 0) s->median = med;
}

__global__ void __launch_bounds__(ML_T, 2) k_median_reset(const double* __restrict__ e, size_t n, const EnergyStats* s, int half,
                                                        ResetPlanes rp) {
  grid_dep_wait();
  const EnergyStats::Half& P = s->half[half];
  if (median_skips(P.lo, P.hi, P.nan != 0)) return;
  const double thr = 1e-9 * s->median + 1e-30;
  const size_t i0 = blockIdx.x * (size_t)ML_T + threadIdx.x, step = (size_t)gridDim.x * ML_T;
  double2 v[ML_E];
  load_energies(e, n, i0, step, v);
  each_energy(e, n, i0, step, v, [&](double x, size_t p) {
    if (!(x > thr)) reset_pixel(rp, n, p);
  });
}

void launch_energy_stats_init(EnergyStats* stats, unsigned long long* scratch, cudaStream_t st) {
  OFC_CUDA(cudaMemsetAsync(scratch, 0, ML_BINS * sizeof(unsigned), st));
  OFC_LAUNCH(k_stats_init, 1, 1, 0, st, stats);
}

void launch_median_reset(const double* energy, size_t n, EnergyStats* stats, int half, bool force,
                         unsigned long long* scratch, const double* ux_in, const double* uy_in, double* ux, double* uy,
                         double* resid, double* slope, cudaStream_t st) {
  const ResetPlanes rp{ux_in, uy_in, ux, uy, resid, slope};
  const int f = force ? 1 : 0;
  if (n <= MED_CLUSTER_N) {
    OFC_LAUNCH_PDL(k_median_cluster, MC_B, MC_T, 0, st, energy, (unsigned)n, stats, f, rp);
    return;
  }
  const unsigned g = median_blocks(n);
  OFC_LAUNCH_PDL(k_median_range, g, ML_T, 0, st, energy, n, stats, half);
  unsigned* hist = (unsigned*)scratch;
  unsigned long long* cand = scratch + ML_BINS / 2;  // after the histogram
  OFC_LAUNCH_PDL(k_median_hist, g, ML_T, 0, st, energy, n, stats, half, f, hist);
  OFC_LAUNCH_PDL(k_median_select, g, ML_T, 0, st, energy, n, stats, half, f, cand);
  if (ux) OFC_LAUNCH_PDL(k_median_reset, g, ML_T, 0, st, energy, n, stats, half, rp);
}

// ---------------------------------------------------------------- confidence
__global__ void k_confidence(const double* __restrict__ energy, const double* __restrict__ resid,
                             const double* __restrict__ ux, const double* __restrict__ uy, int W, int H,
                             const EnergyStats* s, double tol, double conf_min, int border, double B,
                             float* conf_out, double* conf64, uint8_t* low, int* count_low) {
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  size_t p = (size_t)y * W + x;
  double scale = 0.25 * s->median + 1e-30;
  double ratio = energy[p] / scale;
  double tex = ratio != ratio ? ratio : fmin(1.0, ratio);
  double q = resid[p] / tol;
  double c = tex * exp(-(q * q));
  if (border) {
    double tx = x + ux[p], ty = y + uy[p];
    double own = (double)min(min(x, y), min(W - 1 - x, H - 1 - y));
    bool rep = own >= B && tx >= B && ty >= B && (W - 1) - tx >= B && (H - 1) - ty >= B;
    c = rep ? (c != c ? c : fmin(fmax(c, 0.0), 1.0)) : 0.0;
  }
  bool lw = c < conf_min;
  if (conf_out) conf_out[p] = (float)c;
  if (conf64) conf64[p] = c;
  if (low) low[p] = lw ? 1 : 0;
  if (count_low) {
    unsigned m = __ballot_sync(__activemask(), lw);
    if ((threadIdx.x & 31) == __ffs(__activemask()) - 1 && m) atomicAdd(count_low, __popc(m));
  }
}

void launch_confidence(const double* energy, const double* resid, const double* ux, const double* uy, int W, int H,
                       const EnergyStats* stats, double phase_tol, double conf_min, bool border, double B,
                       float* conf_out, double* conf64, uint8_t* low, int* count_low, cudaStream_t st) {
  dim3 g(div_up(W, 128), H);
  OFC_LAUNCH(k_confidence, g, 128, 0, st, energy, resid, ux, uy, W, H, stats, phase_tol, conf_min, border ? 1 : 0, B,
             conf_out, conf64, low, count_low);
}

// ---------------------------------------------------------------- bounded distance tests
// vertical distance (rows) to the nearest src pixel of the column within `cap`, else cap + 1
__global__ void k_vdist(const uint8_t* __restrict__ src, int W, int H, int cap, int* __restrict__ vd,
                        const int* gate) {
  if (gate && *gate == 0) return;
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  int best = cap + 1;
  for (int d = 0; d <= cap && d < best; d++) {
    if ((y - d >= 0 && src[(size_t)(y - d) * W + x]) || (y + d < H && src[(size_t)(y + d) * W + x])) best = d;
  }
  vd[(size_t)y * W + x] = best;
}

// squared distance from vd within cap; mode 0: out |= (d <= limit); mode 1: out = (d > limit); counts ok
__global__ void k_within(const int* __restrict__ vd, int W, int H, int cap, double limit, int mode, uint8_t* out,
                         const int* gate, int* count) {
  if (gate && *gate == 0) return;
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  long best = -1;
  const int* row = vd + (size_t)y * W;
  for (int dx = -cap; dx <= cap; dx++) {
    int xx = x + dx;
    if (xx < 0 || xx >= W) continue;
    int v = row[xx];
    if (v > cap) continue;
    long d2 = (long)dx * dx + (long)v * v;
    if (best < 0 || d2 < best) best = d2;
  }
  bool inside = best >= 0 && sqrt((double)best) <= limit;
  size_t p = (size_t)y * W + x;
  if (mode == 0) {
    if (inside) out[p] = 1;
  } else {
    bool okp = !inside;
    out[p] = okp ? 1 : 0;
    if (count) {
      unsigned m = __ballot_sync(__activemask(), okp);
      if ((threadIdx.x & 31) == __ffs(__activemask()) - 1 && m) atomicAdd(count, __popc(m));
    }
  }
}

// The same test in one pass through a shared-memory tile of WT_X x WT_Y pixels with a halo of cap (<= WT_CAPMAX)
// on every side: the vertical distances of the tile's columns come from two running scans per column (the last
// src row at or above, the next at or below), then each pixel takes the smallest dx^2 + v^2 over |dx| <= cap.
// Results equal k_vdist + k_within's; count (mode 1) is summed per block.
constexpr int WT_X = 128, WT_Y = 32, WT_CAPMAX = 32, WT_T = 256;

template <int CAPT>
__global__ void __launch_bounds__(WT_T) k_within_tile(const uint8_t* __restrict__ src, int W, int H, int cap_rt,
                                                      double limit, int mode, uint8_t* out, const int* gate,
                                                      int* count) {
  grid_dep_wait();
  if (gate && *gate == 0) return;
  const int cap = CAPT ? CAPT : cap_rt;
  __shared__ uint8_t s[(WT_Y + 2 * WT_CAPMAX) * (WT_X + 2 * WT_CAPMAX)];
  __shared__ uint8_t vd[WT_Y * (WT_X + 2 * WT_CAPMAX)];
  __shared__ int wsum[WT_T / 32];
  const int TW = WT_X + 2 * cap, TH = WT_Y + 2 * cap, tid = threadIdx.x;
  const int bx = blockIdx.x * WT_X, by = blockIdx.y * WT_Y;
  // the tile, 8 loads in flight per thread
  for (int i0 = 0; i0 < TW * TH; i0 += 8 * WT_T) {
    uint8_t v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + u * WT_T + tid;
      const int ty = i / TW, tx = i - ty * TW, gx = bx - cap + tx, gy = by - cap + ty;
      v[u] = (i < TW * TH && gx >= 0 && gx < W && gy >= 0 && gy < H) ? __ldg(src + (size_t)gy * W + gx) : 0;
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + u * WT_T + tid;
      if (i < TW * TH) s[i] = v[u];
    }
  }
  __syncthreads();
  for (int tx = tid; tx < TW; tx += WT_T) {
    int last = -(1 << 20);
    for (int ty = 0; ty < cap + WT_Y; ty++) {
      if (s[ty * TW + tx]) last = ty;
      if (ty >= cap) vd[(ty - cap) * TW + tx] = (uint8_t)min(ty - last, cap + 1);
    }
    int next = 1 << 20;
    for (int ty = TH - 1; ty >= cap; ty--) {
      if (s[ty * TW + tx]) next = ty;
      if (ty < cap + WT_Y) {
        uint8_t& v = vd[(ty - cap) * TW + tx];
        v = (uint8_t)min((int)v, min(next - ty, cap + 1));
      }
    }
  }
  __syncthreads();
  int cnt = 0;
  for (int i = tid; i < WT_X * WT_Y; i += WT_T) {  // the same trip count for every thread
    const int r = i / WT_X, c = i - r * WT_X, gx = bx + c, gy = by + r;
    const uint8_t* row = vd + r * TW + c + cap;
    int best = 1 << 30;  // no vertical distance within cap: d2 stays above every limit^2 with limit < cap
#pragma unroll
    for (int dx = -cap; dx <= cap; dx++) {
      const int v = row[dx];
      const int d2 = v > cap ? (1 << 30) : dx * dx + v * v;
      best = min(best, d2);
    }
    const bool inside = best < (1 << 30) && sqrt((double)best) <= limit;
    if (gx < W && gy < H) {
      const size_t p = (size_t)gy * W + gx;
      if (mode == 0) {
        if (inside) out[p] = 1;
      } else {
        out[p] = inside ? 0 : 1;
        cnt += inside ? 0 : 1;
      }
    }
  }
  if (count) {
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((tid & 31) == 0) wsum[tid >> 5] = cnt;
    __syncthreads();
    if (tid == 0) {
      int t = 0;
      for (int w = 0; w < WT_T / 32; w++) t += wsum[w];
      if (t) atomicAdd(count, t);
    }
  }
}

// out |= (distance to src <= limit) (mode 0), or out = (distance > limit) with the count of such pixels (mode 1),
// gated on *gate != 0 when gate is given
static void within(const uint8_t* src, int W, int H, double limit, int mode, uint8_t* out, int* vdist, const int* gate,
                   int* count, cudaStream_t st) {
  const int cap = (int)floor(limit) + 1;
  if (cap <= WT_CAPMAX) {
    dim3 g(div_up(W, WT_X), div_up(H, WT_Y));
    if (cap == 13)  // the default radii (12.22 px)
      OFC_LAUNCH_PDL(k_within_tile<13>, g, WT_T, 0, st, src, W, H, cap, limit, mode, out, gate, count);
    else
      OFC_LAUNCH_PDL(k_within_tile<0>, g, WT_T, 0, st, src, W, H, cap, limit, mode, out, gate, count);
    return;
  }
  dim3 g(div_up(W, 128), H);
  OFC_LAUNCH(k_vdist, g, 128, 0, st, src, W, H, cap, vdist, gate);
  OFC_LAUNCH(k_within, g, 128, 0, st, vdist, W, H, cap, limit, mode, out, gate, count);
}

void launch_within(const uint8_t* src, int W, int H, double limit, int mode, uint8_t* out, int* vdist, cudaStream_t st) {
  within(src, W, H, limit, mode, out, vdist, nullptr, nullptr, st);
}

// ---------------------------------------------------------------- trusted pre-warp
// Nearest ok pixel of each pixel's column (ties to the smaller row): col_d2 = dy^2 (or -1 without one), col_row.
// Two levels: k_col_segments records, per column and segment of CSEG rows, the first and last ok row; each pixel
// then scans its own segment and, beyond it, the segments' summaries (at most H / CSEG of them).
constexpr int CSEG = 64;

__global__ void k_col_segments(const uint8_t* __restrict__ ok, int W, int H, const PrewarpCounts* c,
                               int* __restrict__ seg_first, int* __restrict__ seg_last) {
  grid_dep_wait();
  if (!(c->low > 0 && c->ok > 0 && c->ok < W * H)) return;
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int sg = blockIdx.y;
  if (x >= W) return;
  int y0 = sg * CSEG, y1 = min(H, y0 + CSEG);
  int first = -1, last = -1;
  for (int y = y0; y < y1; y++)
    if (ok[(size_t)y * W + x]) {
      if (first < 0) first = y;
      last = y;
    }
  seg_first[(size_t)sg * W + x] = first;
  seg_last[(size_t)sg * W + x] = last;
}

__global__ void k_col_nearest(const uint8_t* __restrict__ ok, int W, int H, const PrewarpCounts* c,
                              const int* __restrict__ seg_first, const int* __restrict__ seg_last,
                              int* __restrict__ col_d2, int* __restrict__ col_row) {
  grid_dep_wait();
  if (!(c->low > 0 && c->ok > 0 && c->ok < W * H)) return;
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  const size_t p = (size_t)y * W + x;
  const int sg = y / CSEG, y0 = sg * CSEG, y1 = min(H, y0 + CSEG);
  int up = -1, dn = -1;
  for (int yy = y; yy >= y0; yy--)
    if (ok[(size_t)yy * W + x]) { up = yy; break; }
  if (up < 0)
    for (int s2 = sg - 1; s2 >= 0; s2--) {
      int l = seg_last[(size_t)s2 * W + x];
      if (l >= 0) { up = l; break; }
    }
  for (int yy = y; yy < y1; yy++)
    if (ok[(size_t)yy * W + x]) { dn = yy; break; }
  if (dn < 0) {
    const int nseg = (H + CSEG - 1) / CSEG;
    for (int s2 = sg + 1; s2 < nseg; s2++) {
      int f = seg_first[(size_t)s2 * W + x];
      if (f >= 0) { dn = f; break; }
    }
  }
  int r = up;
  long d = up >= 0 ? (long)(y - up) : -1;
  if (dn >= 0 && (r < 0 || (long)(dn - y) < d)) { r = dn; d = dn - y; }
  col_row[p] = r;
  col_d2[p] = r < 0 ? -1 : (int)(d * d);
}

// for every pixel that is not ok: the nearest ok pixel (smallest (d^2, column, row)), then the first-order
// extrapolation u(N) + grad u(N) (X - N) (phaseflow.py:346-354); ok pixels keep u
__global__ void k_extrapolate(const uint8_t* __restrict__ ok, const int* __restrict__ col_d2,
                              const int* __restrict__ col_row, const double* __restrict__ ux,
                              const double* __restrict__ uy, const double* __restrict__ slope, int W, int H,
                              const PrewarpCounts* c, double* ux_pre, double* uy_pre) {
  grid_dep_wait();
  int x = blockIdx.x * blockDim.x + threadIdx.x;
  int y = blockIdx.y;
  if (x >= W) return;
  size_t p = (size_t)y * W + x;
  const bool apply = c->low > 0 && c->ok > 0 && c->ok < W * H;
  if (!apply || ok[p]) {
    ux_pre[p] = ux[p];
    uy_pre[p] = uy[p];
    return;
  }
  const int* cd = col_d2 + (size_t)y * W;
  const int* cr = col_row + (size_t)y * W;
  long best = -1;
  int bc = -1;
  for (long D = 0; D < W; D++) {
    if (best >= 0 && D * D > best) break;
    long xl = x - D, xr = x + D;
    if (xl >= 0 && cd[xl] >= 0) {
      long d2 = D * D + cd[xl];
      if (best < 0 || d2 < best || (d2 == best && xl < bc)) { best = d2; bc = (int)xl; }
    }
    if (D > 0 && xr < W && cd[xr] >= 0) {
      long d2 = D * D + cd[xr];
      if (best < 0 || d2 < best || (d2 == best && xr < bc)) { best = d2; bc = (int)xr; }
    }
  }
  int br = cr[bc];
  size_t q = (size_t)br * W + bc;
  size_t N = (size_t)W * H;
  double dx = (double)x - bc, dy = (double)y - br;
  ux_pre[p] = ux[q] + slope[q] * dx + slope[2 * N + q] * dy;
  uy_pre[p] = uy[q] + slope[N + q] * dx + slope[3 * N + q] * dy;
}

__global__ void k_zero_counts(PrewarpCounts* c) { c->ok = 0; }

void launch_prewarp_fill(const uint8_t* low, const double* ux, const double* uy, const double* slope, int W, int H,
                         double R, PrewarpCounts* counts, uint8_t* ok, int* vdist, int* col_d2, int* col_row,
                         double* ux_pre, double* uy_pre, cudaStream_t st) {
  dim3 g(div_up(W, 128), H);
  OFC_LAUNCH(k_zero_counts, 1, 1, 0, st, counts);
  // ok = distance to the nearest low pixel > R (gated on any low pixel)
  within(low, W, H, R, 1, ok, vdist, (const int*)&counts->low, &counts->ok, st);
  int* seg = vdist;  // the vertical distances are spent: 2 * ceil(H / CSEG) * W ints of segment summaries
  const int nseg = (H + CSEG - 1) / CSEG;
  OFC_LAUNCH_PDL(k_col_segments, dim3(div_up(W, 128), nseg), 128, 0, st, ok, W, H, counts, seg, seg + (size_t)nseg * W);
  OFC_LAUNCH_PDL(k_col_nearest, g, 128, 0, st, ok, W, H, counts, seg, seg + (size_t)nseg * W, col_d2, col_row);
  OFC_LAUNCH_PDL(k_extrapolate, g, 128, 0, st, ok, col_d2, col_row, ux, uy, slope, W, H, counts, ux_pre, uy_pre);
}

// ---------------------------------------------------------------- conversions
__global__ void k_d2f(const double* in, float* out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = (float)in[i];
}
__global__ void k_f2d(const float* in, double* out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = (double)in[i];
}
__global__ void k_fill(double* p, double v, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}
void launch_f64_to_f32(const double* in, float* out, size_t n, cudaStream_t st) {
  OFC_LAUNCH(k_d2f, std::min<size_t>(div_up(n, 256), 4096), 256, 0, st, in, out, n);
}
void launch_f32_to_f64(const float* in, double* out, size_t n, cudaStream_t st) {
  OFC_LAUNCH(k_f2d, std::min<size_t>(div_up(n, 256), 4096), 256, 0, st, in, out, n);
}
void launch_fill_f64(double* p, double v, size_t n, cudaStream_t st) {
  OFC_LAUNCH(k_fill, std::min<size_t>(div_up(n, 256), 4096), 256, 0, st, p, v, n);
}

}  // namespace ofc
