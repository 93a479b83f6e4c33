// common.cuh -- shared device helpers of the optflow B200 engine (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/optflow_cuda.h"

namespace ofc {

constexpr double PI = 3.14159265358979323846;
constexpr int PAD = 32;                 // reflect padding of the Gabor responses (phaseflow.py:47)
constexpr double APERTURE_TOL = 1e-3;   // phaseflow.py:50
constexpr int HORIZON = 21;             // ceil(log(1e-12) / log|sqrt(3) - 2|) (interp.py:10)
constexpr int IIR_WARM = 28;            // samples of warm-up of a segmented recursive filter: z^29 < 3e-17

// An error that leaves the call with a status and a message (EngineError of the reference).
struct Error : std::runtime_error {
  int status;
  Error(int s, const std::string& m) : std::runtime_error(m), status(s) {}
};

#define OFC_CUDA(call)                                                                          \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess)                                                                      \
      throw ::ofc::Error(OFC_ERR_DEVICE, std::string("CUDA error ") + cudaGetErrorString(e_) + \
                                             " at " + __FILE__ + ":" + std::to_string(__LINE__)); \
  } while (0)

// A host-to-device copy that has ended on return. cudaMemcpy of pageable memory returns once the data are staged, before
// they are all on the device, and work on the lanes' streams (which do not wait for the default stream) could read what was
// there before.
inline void upload_now(void* dst, const void* src, size_t bytes) {
  OFC_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
  OFC_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
}

// kernel launch with error check, the engine's launch counter and, in profile mode, CUDA events around the
// launches whose kernel name matches the profile filter (the reference's per-kernel GPU timing,
// OPTFLOW_GPU_KERNELS, rust/README.md:157-159)
struct Profiler;
extern thread_local uint64_t* g_launch_counter;
extern thread_local Profiler* g_profiler;
void prof_before(const char* name, cudaStream_t st, void** token);
void prof_after(void* token, cudaStream_t st);
#define OFC_LAUNCH(kernel, grid, block, smem, stream, ...)                         \
  do {                                                                             \
    void* ofc_tok_ = nullptr;                                                      \
    if (::ofc::g_profiler) ::ofc::prof_before(#kernel, (stream), &ofc_tok_);       \
    kernel<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__);                    \
    OFC_CUDA(cudaGetLastError());                                                  \
    if (ofc_tok_) ::ofc::prof_after(ofc_tok_, (stream));                           \
    if (::ofc::g_launch_counter) ++*::ofc::g_launch_counter;                       \
  } while (0)

// The same with a programmatic dependency on what the stream ran last (where that is a kernel; else an ordinary one): the
// launch is prepared while that kernel drains, and its blocks wait in grid_dep_wait, which every kernel launched this way
// calls before it touches memory, until that kernel has ended and its writes are visible. For the refinement's kernels,
// some 150 dependent launches that small images wait for: 128^2 pairs 1.246 -> 1.216 ms, 256^2 1.588 -> 1.533 ms, 333 x
// 191 2.198 -> 2.126 ms, from 512^2 up 0.2 to 1 %. No kernel releases its dependents early: their waiting blocks would
// take its place on the SMs (2048^2: 30.3 -> 30.7 ms).
#define OFC_LAUNCH_PDL(kernel, grid, block, smem, stream_, ...)                    \
  do {                                                                             \
    void* ofc_tok_ = nullptr;                                                      \
    if (::ofc::g_profiler) ::ofc::prof_before(#kernel, (stream_), &ofc_tok_);      \
    cudaLaunchConfig_t ofc_cfg_{};                                                 \
    ofc_cfg_.gridDim = (grid);                                                     \
    ofc_cfg_.blockDim = (block);                                                   \
    ofc_cfg_.dynamicSmemBytes = (smem);                                            \
    ofc_cfg_.stream = (stream_);                                                   \
    cudaLaunchAttribute ofc_at_{};                                                 \
    ofc_at_.id = cudaLaunchAttributeProgrammaticStreamSerialization;               \
    ofc_at_.val.programmaticStreamSerializationAllowed = 1;                        \
    ofc_cfg_.attrs = &ofc_at_;                                                     \
    ofc_cfg_.numAttrs = 1;                                                         \
    cudaLaunchKernelEx(&ofc_cfg_, kernel, __VA_ARGS__);                            \
    OFC_CUDA(cudaGetLastError());                                                  \
    if (ofc_tok_) ::ofc::prof_after(ofc_tok_, (stream_));                          \
    if (::ofc::g_launch_counter) ++*::ofc::g_launch_counter;                       \
  } while (0)
// the first statement of every kernel launched by OFC_LAUNCH_PDL, on every thread (a later kernel's wait then covers the
// earlier ones'); an ordinary launch passes it at once
__device__ __forceinline__ void grid_dep_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

inline unsigned div_up(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

// raises kernel fn's dynamic shared-memory limit on the current device to at least `bytes` and never lowers it:
// the limit belongs to the kernel, not to a launch, so host threads that launch it with different sizes at once
// (the pair driver's lanes) must not shrink it under each other's launches
void raise_smem_limit(const void* fn, size_t bytes);

// two float32 values in a 64-bit register pair; fma on both halves in one instruction, each rounded as fmaf
__device__ __forceinline__ unsigned long long f32x2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f32x2_split(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long mul_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// atan2(y, x) in float32 for finite or NaN arguments, from the mathematics: with a = min(|x|, |y|) / max(|x|, |y|)
// in [0, 1], atan(a) = a P(a^2), P the 8-term fit of atan(a) / a made by atan_fit.py (a minimax fit of the relative
// error by iteratively reweighted least squares; 1.6e-7 rad at most in a float32 Horner); then pi/2 - r where
// |y| > |x|, pi - r where x is negative (its sign bit: -0 included) and the sign of y (+-0 as atan2 gives them).
// At most 5e-7 rad (about 2 ulp of pi) from the exact angle of the float32 arguments with the quotient's rounding and
// the reflections; NaN in gives NaN; atan2(+-0, +0) = +-0 and atan2(+-0, -0) = +-pi. The quotient is the fast one in
// the reciprocal's range, the rounded one where the larger magnitude is outside (1e-30, 1e30).
__device__ __forceinline__ bool atan2_fast(float mx) { return mx > 1e-30f && mx < 1e30f; }
__device__ __forceinline__ float atan2_ratio(float ax, float ay) {
  const float mx = fmaxf(ax, ay), mn = fminf(ax, ay);
  if (atan2_fast(mx)) return __fdividef(mn, mx);
  return mx > 0.f ? mn / mx : 0.f;
}
// the rounded quotient by the float64 reciprocal and two Newton-Raphson steps (r + r (1 - d r)), without the call that
// mn / mx takes: in the accumulate's loop, where no usual value reaches it, a call costs 8 % of the kernel (0.513 against
// 0.472 ms at 2048^2) by its register convention alone. The product is within 2^-51 of the quotient before its one rounding
// to float32. NaN where both are
__device__ __forceinline__ float atan2_ratio_far(float mn, float mx) {
  const double d = (double)mx;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(fma(-d, r, 1.0), r, r);
  r = fma(fma(-d, r, 1.0), r, r);
  const float q = (float)((double)mn * r);
  if (mx > 3.4028234e38f) return mn > 3.4028234e38f ? mn - mx : 0.f;  // infinite: NaN or 0
  return mx == 0.f ? 0.f : q;
}
// r = atan(min / max) reflected into the argument's octant
__device__ __forceinline__ float atan2_octant(float r, float x, float y) {
  if (fabsf(y) > fabsf(x)) r = 1.57079632679489662f - r;
  if (signbit(x)) r = 3.14159265358979324f - r;
  return copysignf(r, y);
}
__device__ __forceinline__ float atan2_phase(float y, float x) {
  const float a = atan2_ratio(fabsf(x), fabsf(y));
  const float t = a * a;
  float p = -4.693272372e-03f;
  p = fmaf(p, t, 2.425239656e-02f);
  p = fmaf(p, t, -5.948639446e-02f);
  p = fmaf(p, t, 9.914293821e-02f);
  p = fmaf(p, t, -1.401948170e-01f);
  p = fmaf(p, t, 1.996972415e-01f);
  p = fmaf(p, t, -3.333199078e-01f);
  p = fmaf(p, t, 9.999999010e-01f);
  const float r = atan2_octant(p * a, x, y);
  return (y != y || x != x) ? y + x : r;
}
// atan2_phase of two arguments with the polynomial of both in packed instructions: the same value for numbers. Where one
// argument is NaN and the other finite it may give any angle: the caller's r1 or r2 is NaN then, and with its weight
// |r1| |r2| every sum (products that overflow leave the other argument infinite or NaN, which gives NaN here too)
__device__ __forceinline__ void atan2_phase_pair(float y0, float x0, float y1, float x1, float& r0, float& r1) {
  const float mx0 = fmaxf(fabsf(x0), fabsf(y0)), mn0 = fminf(fabsf(x0), fabsf(y0));
  const float mx1 = fmaxf(fabsf(x1), fabsf(y1)), mn1 = fminf(fabsf(x1), fabsf(y1));
  float a0 = __fdividef(mn0, mx0), a1 = __fdividef(mn1, mx1);
  if (!atan2_fast(mx0)) a0 = atan2_ratio_far(mn0, mx0);
  if (!atan2_fast(mx1)) a1 = atan2_ratio_far(mn1, mx1);
  const unsigned long long a = f32x2(a0, a1);
  const unsigned long long t = mul_f32x2(a, a);
  unsigned long long p = f32x2(-4.693272372e-03f, -4.693272372e-03f);
  p = fma_f32x2(p, t, f32x2(2.425239656e-02f, 2.425239656e-02f));
  p = fma_f32x2(p, t, f32x2(-5.948639446e-02f, -5.948639446e-02f));
  p = fma_f32x2(p, t, f32x2(9.914293821e-02f, 9.914293821e-02f));
  p = fma_f32x2(p, t, f32x2(-1.401948170e-01f, -1.401948170e-01f));
  p = fma_f32x2(p, t, f32x2(1.996972415e-01f, 1.996972415e-01f));
  p = fma_f32x2(p, t, f32x2(-3.333199078e-01f, -3.333199078e-01f));
  p = fma_f32x2(p, t, f32x2(9.999999010e-01f, 9.999999010e-01f));
  f32x2_split(mul_f32x2(p, a), r0, r1);
  r0 = atan2_octant(r0, x0, y0);
  r1 = atan2_octant(r1, x1, y1);
}

// ---------------------------------------------------------------- cubic B-spline (interp.py)
__host__ __device__ inline long mirror_idx(long i, long n) {  // interp.py:38-43
  if (n == 1) return 0;
  long p = 2 * (n - 1);
  i = i < 0 ? -i : i;
  i %= p;
  return i >= n ? p - i : i;
}

// the reference's quotients by 6 as products with the nearest double to 1/6: a float64 division is a sequence of a
// dozen dependent instructions on the GPU, and the product is within an ulp of the quotient
__host__ __device__ inline void bspline_weights(double t, double w[4]) {  // interp.py:46-49
  const double s = 1.0 / 6.0;
  double t2 = t * t, t3 = t2 * t;
  double u = 1 - t;
  w[0] = u * u * u * s;
  w[1] = (3 * t3 - 6 * t2 + 4) * s;
  w[2] = (-3 * t3 + 3 * t2 + 3 * t + 1) * s;
  w[3] = t3 * s;
}

// taps of sample(): clamp to [0, n-1], floor, weights, mirrored indices (interp.py:52-69)
struct Taps {
  int xi[4], yi[4];
  double wx[4], wy[4];
  bool cx;  // xi[k] = xi[0] + k (no reflection in x): a row's four taps are adjacent
};

// mirror_idx for an index at most one reflection outside [0, n) (the taps of a clamped position lie in
// [-1, n + 1]): two compares instead of a division; the general rule where one reflection is not enough (n < 3)
__device__ __forceinline__ int mirror_near(int i, int n) {
  int m = i < 0 ? -i : i;
  if (m >= n) m = 2 * (n - 1) - m;
  if (m < 0 || m >= n) m = (int)mirror_idx(i, n);
  return m;
}

__device__ inline bool make_taps(double x, double y, int w, int h, Taps& t) {
  if (!(x == x) || !(y == y)) return false;
  x = fmin(fmax(x, 0.0), (double)(w - 1));
  y = fmin(fmax(y, 0.0), (double)(h - 1));
  double fx = floor(x), fy = floor(y);
  int x0 = (int)fx, y0 = (int)fy;
  bspline_weights(x - fx, t.wx);
  bspline_weights(y - fy, t.wy);
  // taps inside the plane (the usual case) need no mirroring: the same indices without the reflection tests
  const bool ix = x0 >= 1 && x0 + 2 <= w - 1, iy = y0 >= 1 && y0 + 2 <= h - 1;
  t.cx = ix;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    t.xi[k] = ix ? x0 + k - 1 : mirror_near(x0 + k - 1, w);
    t.yi[k] = iy ? y0 + k - 1 : mirror_near(y0 + k - 1, h);
  }
  return true;
}

template <class T>
__device__ inline double sample_real(const T* c, int w, const Taps& t) {
  double out = 0;
  if (t.cx) {  // adjacent taps: one address per row, the same operations in the same order
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const T* row = c + (size_t)t.yi[j] * w + t.xi[0];
      double acc = t.wx[0] * (double)row[0];
#pragma unroll
      for (int k = 1; k < 4; k++) acc += t.wx[k] * (double)row[k];
      out += t.wy[j] * acc;
    }
    return out;
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const T* row = c + (size_t)t.yi[j] * w;
    double acc = t.wx[0] * (double)row[t.xi[0]];
#pragma unroll
    for (int k = 1; k < 4; k++) acc += t.wx[k] * (double)row[t.xi[k]];
    out += t.wy[j] * acc;
  }
  return out;
}

// two real splines sampled at the same taps (one set of 32-bit offsets for both)
template <class T>
__device__ __forceinline__ void sample2_real(const T* __restrict__ c1, const T* __restrict__ c2, int w, const Taps& t,
                                             double& o1, double& o2) {
  int o[16];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int k = 0; k < 4; k++) o[j * 4 + k] = t.yi[j] * w + t.xi[k];
  o1 = 0;
  o2 = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    double a1 = t.wx[0] * (double)c1[o[j * 4]], a2 = t.wx[0] * (double)c2[o[j * 4]];
#pragma unroll
    for (int k = 1; k < 4; k++) {
      a1 += t.wx[k] * (double)c1[o[j * 4 + k]];
      a2 += t.wx[k] * (double)c2[o[j * 4 + k]];
    }
    o1 += t.wy[j] * a1;
    o2 += t.wy[j] * a2;
  }
}

// two real splines stored interleaved (double2 per pixel), sampled at the same taps
__device__ __forceinline__ double2 sample_pair(const double2* __restrict__ c, int w, const Taps& t) {
  double o1 = 0, o2 = 0;
  if (t.cx) {  // adjacent taps: one address per row, the four loads at fixed offsets from it
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const double2* row = c + (size_t)t.yi[j] * w + t.xi[0];
      const double2 c0 = __ldg(row);
      double a1 = t.wx[0] * c0.x, a2 = t.wx[0] * c0.y;
#pragma unroll
      for (int k = 1; k < 4; k++) {
        const double2 v = __ldg(row + k);
        a1 += t.wx[k] * v.x;
        a2 += t.wx[k] * v.y;
      }
      o1 += t.wy[j] * a1;
      o2 += t.wy[j] * a2;
    }
    return make_double2(o1, o2);
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const double2* row = c + (size_t)t.yi[j] * w;
    const double2 c0 = __ldg(row + t.xi[0]);
    double a1 = t.wx[0] * c0.x, a2 = t.wx[0] * c0.y;
#pragma unroll
    for (int k = 1; k < 4; k++) {
      const double2 v = __ldg(row + t.xi[k]);
      a1 += t.wx[k] * v.x;
      a2 += t.wx[k] * v.y;
    }
    o1 += t.wy[j] * a1;
    o2 += t.wy[j] * a2;
  }
  return make_double2(o1, o2);
}

// complex spline stored as float2; float accumulation of the 16 taps with f64-derived weights
__device__ inline float2 sample_c32(const float2* __restrict__ c, int w, const Taps& t) {
  float re = 0.f, im = 0.f;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float2* row = c + (size_t)t.yi[j] * w;
    float are = 0.f, aim = 0.f;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      float2 v = __ldg(row + t.xi[k]);
      float wk = (float)t.wx[k];
      are = fmaf(wk, v.x, are);
      aim = fmaf(wk, v.y, aim);
    }
    float wj = (float)t.wy[j];
    re = fmaf(wj, are, re);
    im = fmaf(wj, aim, im);
  }
  return make_float2(re, im);
}

// scalar bspline prefilter pole
__host__ __device__ inline double bspline_z() { return sqrt(3.0) - 2.0; }  // interp.py:9

// one blob of the synthetic speckle renderer (synth.cu): reference centre, radius, amplitude and the subsample
// rectangle [i0, i1) x [j0, j1) it adds to
struct SynthBlob {
  double cx, cy, r, a;
  int i0, i1, j0, j1;
};

}  // namespace ofc
