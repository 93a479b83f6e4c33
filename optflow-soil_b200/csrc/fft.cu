// fft.cu -- FP32 mixed-radix FFTs in shared memory with the fused Gabor multiply and B-spline prefilter.
//
// One thread block transforms C interleaved lines held in shared memory (element i of line l at
// buf[i * C + l]), ping-ponging between two buffers of L * C values: each Stockham stage reads a butterfly's
// inputs from one and writes its outputs to the other. Radices 2, 4 and 8 have register butterflies, 3, 5, 7,
// 11, 13, 17 and 19 the symmetric odd form, 23, 29 and 31 a direct DFT. Twiddles come from a table rounded from
// float64.
//
// The pass structure of one "responses" evaluation (per outer iteration of the fine stage):
//   rows:    reflect pad + real->complex + forward row FFT                      (read 4 B/px, write 8 B/px)
//   columns: forward column FFT in place (read 8, write 8); then per (column pair, filter k): x G_k and the
//            B-spline prefilter's periodic factor 1 / ((4 + 2 cos wx)(4 + 2 cos wy)) (separable tables), inverse
//            column FFT, the prefilter's edge terms along y                        (read 8F, write 8F)
//   rows:    inverse row FFT, the prefilter's edge terms along x, scale 36 / (ph pw)  (read 8F, write 8F)
// The prefilter is separable and linear, so its factors and edge terms along one axis commute with the
// transforms along the other, and the result is bspline_coeffs(ifft2(F2 * G)) of phaseflow.py:456 up to rounding.
#include "fft.cuh"

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <type_traits>

#include <cuda_pipeline.h>

namespace ofc {

// ------------------------------------------------------------------------------------------ host
bool fft_supported(int L) {
  if (L < 1) return false;
  int m = L;
  for (int p : {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31})
    while (m % p == 0) m /= p;
  return m == 1;
}

static int stage_count(int m) {
  int n = 0;
  while (m % 8 == 0) { n++; m /= 8; }
  while (m % 4 == 0) { n++; m /= 4; }
  while (m % 2 == 0) { n++; m /= 2; }
  for (int p : {3, 5, 7, 11, 13, 17, 19, 23, 29, 31})
    while (m % p == 0) { n++; m /= p; }
  return n;
}

// The cost of a Bluestein inner length M: M times its Stockham stages of the radices with a butterfly of their own (8,
// 4, 2 and the odd primes up to 19), a stage of radix 11 or 13 counted 1.2 and of 17 or 19 1.5 (their butterflies take
// more registers); infinite for other factors. The transforms are bound by their stage barriers, not by arithmetic:
// 604 = 4 151 (the padded height of 540-row frames) takes M = 1216 = 8 8 19 (3 stages) instead of the smallest
// 2^a 3^b 5^c 7^d, 1215 = 3^5 5 (6 stages).
static double bluestein_cost(int M) {
  double c = 0;
  int m = M;
  while (m % 8 == 0) { c += 1; m /= 8; }
  while (m % 4 == 0) { c += 1; m /= 4; }
  while (m % 2 == 0) { c += 1; m /= 2; }
  for (int p : {3, 5, 7, 11, 13, 17, 19}) {
    const double w = p <= 7 ? 1.0 : (p <= 13 ? 1.2 : 1.5);
    while (m % p == 0) { c += w; m /= p; }
  }
  return m == 1 ? c * M : 1e30;
}

int fft_work_length(int L) {
  if (L < 1) return 0;
  if (fft_supported(L)) return stage_count(L) <= FFT_MAXST ? L : 0;
  // Bluestein: among the lengths M in [2L - 1, 1.25 (2L - 1)] the one of least stage cost (the smallest on ties),
  // never above the smallest 2^a 3^b 5^c 7^d where that one fits the passes' shared memory and a larger one might not
  // (about 6800: four line buffers of the row pass, two two-column buffers of the column pass)
  const int lo = 2 * L - 1;
  int smooth = 0;
  for (int M = lo; M <= 8 * L && !smooth; M++) {
    int m = M;
    for (int p : {2, 3, 5, 7})
      while (m % p == 0) m /= p;
    if (m == 1) smooth = M;
  }
  constexpr int FIT = 6800;
  const int hi = (smooth && smooth <= FIT) ? std::min(lo + lo / 4, std::max(smooth, FIT)) : lo + lo / 4;
  int best = 0;
  double bc = 1e29;  // below the cost of a length with an unsupported factor
  for (int M = lo; M <= hi; M++) {
    const double c = bluestein_cost(M);
    if (c < bc) {
      bc = c;
      best = M;
    }
  }
  return best && stage_count(best) <= FFT_MAXST ? best : 0;
}

std::vector<float2> fft_bluestein_tables(int L, int M) {
  // chirp w[n] = exp(-i pi n^2 / L): the phase from n^2 mod 2L in integers, then float64
  std::vector<double> wr(L), wi(L);
  for (int n = 0; n < L; n++) {
    const long long q = ((long long)n * n) % (2LL * L);
    const double a = -PI * (double)q / (double)L;
    wr[n] = std::cos(a);
    wi[n] = std::sin(a);
  }
  // b = conj(w) wrapped to length M; filt = DFT_M(b) / M in float64 (a direct sum with an integer-indexed table)
  std::vector<double> br(M, 0.0), bi(M, 0.0), cr(M), ci(M);
  for (int n = 0; n < L; n++) {
    br[n] = wr[n];
    bi[n] = -wi[n];
    if (n) {
      br[M - n] = wr[n];
      bi[M - n] = -wi[n];
    }
  }
  for (int t = 0; t < M; t++) {
    const double a = -2.0 * PI * (double)t / (double)M;
    cr[t] = std::cos(a);
    ci[t] = std::sin(a);
  }
  std::vector<float2> out((size_t)L + M);
  for (int n = 0; n < L; n++) out[n] = make_float2((float)wr[n], (float)wi[n]);
  for (int k = 0; k < M; k++) {
    double sr = 0.0, si = 0.0;
    long long idx = 0;
    for (int n = 0; n < M; n++) {
      if (br[n] != 0.0 || bi[n] != 0.0) {
        sr += br[n] * cr[idx] - bi[n] * ci[idx];
        si += br[n] * ci[idx] + bi[n] * cr[idx];
      }
      idx += k;
      if (idx >= M) idx -= M;
    }
    out[(size_t)L + k] = make_float2((float)(sr / M), (float)(si / M));
  }
  return out;
}

namespace {
std::mutex g_plan_mu;
std::map<int, int> g_plan_table;  // padded length -> factor order (fft_set_plan_variant)
}  // namespace

void fft_set_plan_variant(int L, int variant) {
  std::lock_guard<std::mutex> lk(g_plan_mu);
  if (variant <= 0) g_plan_table.erase(L);
  else g_plan_table[L] = variant;
}

int fft_plan_variant(int L) {
  std::lock_guard<std::mutex> lk(g_plan_mu);
  auto it = g_plan_table.find(L);
  return it == g_plan_table.end() ? 0 : it->second;
}

// The factor orders a plan of length n can take (the transform is the same; the stages, their strides and the
// rounding differ): 0 radix 8 first, then 4, 2 and the odd radices ascending; 1 the odd radices first; 2 the power of
// two in radix-4 stages (a radix 2 last when the power is odd); 3 the order of 0 reversed.
static std::vector<int> factor_order(int n, int variant) {
  std::vector<int> two, odd;
  int m = n, e = 0;
  while (m % 2 == 0) { m /= 2; e++; }
  for (int p : {3, 5, 7, 11, 13, 17, 19, 23, 29, 31})
    while (m % p == 0) { odd.push_back(p); m /= p; }
  if (m != 1) return {};
  if (variant == 2) {
    for (; e >= 2; e -= 2) two.push_back(4);
    if (e) two.push_back(2);
  } else {
    for (; e >= 3; e -= 3) two.push_back(8);
    if (e == 2) two.push_back(4);
    if (e == 1) two.push_back(2);
  }
  std::vector<int> f;
  if (variant == 1) {
    f = odd;
    f.insert(f.end(), two.begin(), two.end());
  } else {
    f = two;
    f.insert(f.end(), odd.begin(), odd.end());
  }
  if (variant == 3) std::reverse(f.begin(), f.end());
  return f;
}

FftPlan fft_make_plan(int L) { return fft_make_plan(L, fft_plan_variant(L)); }

FftPlan fft_make_plan(int L, int variant) {
  const int work = fft_work_length(L);
  if (work == 0) throw Error(OFC_ERR_WINDOW, "no FFT plan for length " + std::to_string(L));
  if (variant < 0 || variant >= FFT_PLAN_VARIANTS) throw Error(OFC_ERR_ARG, "no FFT plan variant " + std::to_string(variant));
  FftPlan pl;
  pl.L = L;
  pl.M = work == L ? 0 : work;
  // the plans fixed at compile time keep the default order
  std::vector<int> f = factor_order(work, fft_fixed_length(work) || work == FFT_FIXED_M ? 0 : variant);
  if (f.empty() || (int)f.size() > FFT_MAXST)
    throw Error(OFC_ERR_WINDOW, "FFT length " + std::to_string(L) + " needs too many stages");
  pl.inner = pl.M && f == factor_order(work, 0) ? work : 0;
  int s = 1;
  pl.nst = (int)f.size();
  for (int i = 0; i < pl.nst; i++) {
    pl.p[i] = f[i];
    pl.s[i] = s;
    // ceil(2^32 / s): q = umulhi(bi, magic) = floor(bi / s) for every bi < L * 4 here
    pl.magic[i] = s == 1 ? 0u : (unsigned)((((unsigned long long)1 << 32) + s - 1) / s);
    s *= f[i];
  }
  for (int i = 0, o = 0; i < pl.nst; i++) {
    pl.so[i] = o;
    o += (pl.p[i] - 1) * (work / (pl.p[i] * pl.s[i]));
  }
  return pl;
}

// W[t] = exp(-2 pi i t / L), t < L, rounded from float64
static std::vector<float2> fft_twiddles(int L) {
  std::vector<float2> t(L);
  for (int i = 0; i < L; i++) {
    double a = -2.0 * PI * (double)i / (double)L;
    t[i] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  return t;
}

std::vector<float2> fft_tables(const FftPlan& pl) {
  const int SL = fft_work_len(pl);
  const std::vector<float2> tw = fft_twiddles(SL);
  std::vector<float2> out;
  for (int i = 0; i < pl.nst; i++) {
    const int m = SL / (pl.p[i] * pl.s[i]);
    for (int k = 1; k < pl.p[i]; k++)
      for (int q = 0; q < m; q++) out.push_back(tw[(size_t)k * q * pl.s[i]]);
  }
  const size_t n = out.size();  // the inverse transform's conjugates
  for (size_t i = 0; i < n; i++) out.push_back(make_float2(out[i].x, -out[i].y));
  if (pl.M) {
    const std::vector<float2> bt = fft_bluestein_tables(pl.L, pl.M);
    out.insert(out.end(), bt.begin(), bt.end());
  }
  return out;
}

void fft_bind(FftPlan& pl, const float2* d) {
  const int SL = fft_work_len(pl);
  pl.stw = d;
  const int last = pl.nst - 1;
  pl.nstw = pl.so[last] + (pl.p[last] - 1) * (SL / (pl.p[last] * pl.s[last]));
  if (pl.M) {
    pl.chirp = pl.stw + 2 * pl.nstw;
    pl.filt = pl.chirp + pl.L;
  }
}

// Threads of a block of a runtime plan that holds `smem` bytes: the count whose blocks finish most lines per time on an SM.
// A block's line takes the longer of its latency (the rounds of butterflies of its stages one after the other, an
// instruction of a lone warp every 6 cycles, a barrier per stage) and its share of the issue slots (2.4 instructions per
// cycle between the resident blocks, as many as shared memory and 80 registers per thread admit). Small transforms get
// several blocks of few threads with little idling in the stages of large radices, a transform that fills shared memory
// by itself many threads (Bluestein's 4096 on a column pair: one block per SM). *cycles: that time per block.
static int rt_threads(const FftPlan& pl, int C, size_t smem, double* cycles = nullptr) {
  const int SL = fft_work_len(pl);
  const int fit = std::max<int>(1, (int)((227 * 1024) / (smem + 1024)));
  int best = 256;
  double bt = 1e300;
  for (int T = 96; T <= RT_T; T += 32) {
    const int blocks = std::min(fit, std::max(1, 65536 / (80 * T)));
    double lat = 0, work = 0;
    for (int i = 0; i < pl.nst; i++) {
      const int P = pl.p[i], sh = P >= 23 ? 4 : 1, nb = sh > 1 ? (SL / P * C + 31) / 32 * 32 * sh : SL / P * C;
      const double c = sh > 1 ? 4.5 * P * P / sh + 30.0 * P : (P % 2 ? (P - 1) * (P - 1) : 8 * P) + 25.0 * P;  // instructions
      lat += (double)((nb + T - 1) / T) * c * 6.0 + 150.0;
      work += (double)nb / 32.0 * c;
    }
    const double t = std::max(lat / blocks, work / 2.4);
    if (t < bt * 0.995) {
      bt = t;
      best = T;
    }
  }
  if (cycles) *cycles = bt;
  return best;
}

int fft_threads(int L, int C) {
  int need = (L * C + FFT_E - 1) / FFT_E;
  int unit = 32;
  while (unit % C) unit += 32;  // multiple of 32 and of C
  int cap = (FFT_TMAX / unit) * unit;
  int T = ((need + unit - 1) / unit) * unit;
  return std::max(unit, std::min(T, cap));
}

size_t gabor_yt2_offset(int ph, int pw, int F) {
  const size_t base = (size_t)4 * (pw + ph) + (size_t)F * (pw + ph);
  return (base + 1) & ~(size_t)1;
}

std::vector<double> gabor_tables_host(int ph, int pw, const ofc_config& c) {
  int F = c.n_scales * c.n_orient;
  std::vector<double> t((size_t)4 * (pw + ph) + (size_t)F * (pw + ph));
  double* fx = t.data();
  double* fy = fx + pw;
  double* hx = fy + ph;
  double* hy = hx + pw;
  double* omx = hy + ph;
  double* omy = omx + pw;
  double* ex = omy + ph;
  double* ey = ex + (size_t)F * pw;
  auto freq = [](int n, double* f) {  // np.fft.fftfreq(n) * 2 * pi
    double val = 1.0 / n;
    int N = (n - 1) / 2 + 1;
    for (int i = 0; i < n; i++) f[i] = (double)(i < N ? i : i - n) * val * 2 * PI;
  };
  freq(pw, fx);
  freq(ph, fy);
  double smax = 0;
  for (int i = 0; i < c.n_scales; i++) smax = std::max(smax, c.scales[i]);
  double s_hp = c.dc_cut * c.lam * smax / (2 * PI);
  for (int x = 0; x < pw; x++) {
    double e = -(fx[x] * fx[x]) * (s_hp * s_hp) / 2;
    hx[x] = std::exp(e);
    omx[x] = -std::expm1(e);
  }
  for (int y = 0; y < ph; y++) {
    double e = -(fy[y] * fy[y]) * (s_hp * s_hp) / 2;
    hy[y] = std::exp(e);
    omy[y] = -std::expm1(e);
  }
  int k = 0;
  for (int si = 0; si < c.n_scales; si++) {
    double w0 = 2 * PI / (c.lam * c.scales[si]);
    double s = c.bandwidth * w0;
    for (int o = 0; o < c.n_orient; o++, k++) {
      double th = PI * o / c.n_orient;
      double cx = w0 * std::cos(th), cy = w0 * std::sin(th);
      for (int x = 0; x < pw; x++) { double d = fx[x] - cx; ex[(size_t)k * pw + x] = std::exp(-(d * d) / (2 * s * s)); }
      for (int y = 0; y < ph; y++) { double d = fy[y] - cy; ey[(size_t)k * ph + y] = std::exp(-(d * d) / (2 * s * s)); }
    }
  }
  // the B-spline prefilter on the periodic grid, per axis: 1 / (4 + 2 cos w)
  double* bx = ey + (size_t)F * ph;
  double* by = bx + pw;
  for (int x = 0; x < pw; x++) bx[x] = 1.0 / (4.0 + 2.0 * std::cos(2 * PI * (double)x / pw));
  for (int y = 0; y < ph; y++) by[y] = 1.0 / (4.0 + 2.0 * std::cos(2 * PI * (double)y / ph));
  // per filter and row: (omy[y], ey_k[y] by[y]), from an even offset (a float2 table in the float32 image)
  std::vector<double> yt((size_t)2 * F * ph);
  for (int k2 = 0; k2 < F; k2++)
    for (int y = 0; y < ph; y++) {
      yt[2 * ((size_t)k2 * ph + y)] = omy[y];
      yt[2 * ((size_t)k2 * ph + y) + 1] = ey[(size_t)k2 * ph + y] * by[y];
    }
  const size_t o = gabor_yt2_offset(ph, pw, F);
  t.resize(o + yt.size(), 0.0);
  std::copy(yt.begin(), yt.end(), t.begin() + o);
  return t;
}

void gabor_bind(GaborTables& g, const double* d64, const float* d32, int ph, int pw, int F) {
  g.F = F;
  g.ph = ph;
  g.pw = pw;
  g.fx = d64;
  g.fy = g.fx + pw;
  g.hx = g.fy + ph;
  g.hy = g.hx + pw;
  g.omx = g.hy + ph;
  g.omy = g.omx + pw;
  g.ex = g.omy + ph;
  g.ey = g.ex + (size_t)F * pw;
  g.hxf = d32 + pw + ph;
  g.omxf = g.hxf + pw + ph;
  g.omyf = g.omxf + pw;
  g.exf = g.omyf + ph;
  g.eyf = g.exf + (size_t)F * pw;
  g.bxf = g.eyf + (size_t)F * ph;
  g.byf = g.bxf + pw;
  g.yt2 = (const float2*)(d32 + gabor_yt2_offset(ph, pw, F));
}

// ------------------------------------------------------------------------------------------ device
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }
// multiply by -i (forward) or +i (inverse)
__device__ __forceinline__ float2 rot(float2 a, bool inv) { return inv ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x); }
template <class C2> __device__ __forceinline__ C2 mkc(double re, double im);
template <> __device__ __forceinline__ float2 mkc<float2>(double re, double im) { return make_float2((float)re, (float)im); }

// cos and sin of 2 pi m / P at compile time (Taylor series after reduction to [-pi/8, pi/8] by octant; exact to
// float64 rounding for the small P here), for the constant coefficients of the odd-radix butterflies
constexpr double ct_poly_sin(double x) {
  double t = x, s = x;
  for (int n = 1; n < 14; n++) {
    t *= -x * x / ((2 * n) * (2 * n + 1));
    s += t;
  }
  return s;
}
constexpr double ct_poly_cos(double x) {
  double t = 1, s = 1;
  for (int n = 1; n < 14; n++) {
    t *= -x * x / ((2 * n - 1) * (2 * n));
    s += t;
  }
  return s;
}
// angle 2 pi m / P = q (pi / 4) + r with |r| <= pi / 8
constexpr void ct_sincos(int m, int P, double& c, double& sn) {
  double a = 2 * PI * (double)m / (double)P;
  int q = (int)(a / (PI / 4) + 0.5);
  double r = a - q * (PI / 4);
  double cr = ct_poly_cos(r), sr = ct_poly_sin(r);
  constexpr double h = 0.70710678118654752440;  // cos(pi / 4)
  double cq[8] = {1, h, 0, -h, -1, -h, 0, h}, sq[8] = {0, h, 1, h, 0, -h, -1, -h};
  c = cq[q & 7] * cr - sq[q & 7] * sr;
  sn = sq[q & 7] * cr + cq[q & 7] * sr;
}
template <int P>
struct OddCoef {  // cs[k][j] = cos(2 pi j k / P), sn[k][j] = -sin(2 pi j k / P) (the forward kernel exp(-2 pi i jk / P))
  float cs[P][P] = {}, sn[P][P] = {};
  constexpr OddCoef() {
    for (int k = 0; k < P; k++)
      for (int j = 0; j < P; j++) {
        double c = 0, s = 0;
        ct_sincos((j * k) % P, P, c, s);
        cs[k][j] = (float)c;
        sn[k][j] = (float)(-s);
      }
  }
};

// Odd-radix butterfly with the symmetric form: for j = 1..(P-1)/2, a_j = v_j + v_{P-j}, b_j = v_j - v_{P-j};
// o_0 = v_0 + sum a_j; o_k = v_0 + sum_j a_j cos_jk + i sum_j b_j sin_jk, o_{P-k} = the same with -i, where
// w^{jk} = cos_jk + i sin_jk (w = exp(-2 pi i / P), conjugated for the inverse) are compile-time constants.
template <int P, class C2, class Load, class Emit>
__device__ __forceinline__ void odd_butterfly(Load in, bool inv, Emit emit) {
  constexpr int Hh = (P - 1) / 2;
  constexpr OddCoef<P> K{};
  C2 v0 = in(0);
  C2 av[Hh], bv[Hh];
#pragma unroll
  for (int j = 1; j <= Hh; j++) {
    C2 x = in(j), y = in(P - j);
    av[j - 1] = cadd(x, y);
    bv[j - 1] = csub(x, y);
  }
  C2 s0 = v0;
#pragma unroll
  for (int j = 0; j < Hh; j++) s0 = cadd(s0, av[j]);
  emit(0, s0);
  const float sg = inv ? -1.f : 1.f;
#pragma unroll
  for (int k = 1; k <= Hh; k++) {
    C2 t = v0, u = mkc<C2>(0.0, 0.0);
#pragma unroll
    for (int j = 1; j <= Hh; j++) {
      const float cs = K.cs[k][j], sn = K.sn[k][j];
      t.x = fmaf(av[j - 1].x, cs, t.x);
      t.y = fmaf(av[j - 1].y, cs, t.y);
      u.x = fmaf(bv[j - 1].x, sn, u.x);
      u.y = fmaf(bv[j - 1].y, sn, u.y);
    }
    u.x *= sg;
    u.y *= sg;
    // i u = (-u.y, u.x)
    emit(k, mkc<C2>(t.x - u.y, t.y + u.x));
    emit(P - k, mkc<C2>(t.x + u.y, t.y - u.x));
  }
}

// Shared-memory layouts of the transform buffers: element i at i + (i >> sh), sh = FFT_PAD (one pad slot
// per 16 values) or 31 (no padding; i < 2^31). A stage whose outputs lie s * C apart with s * C < 32 writes
// padded, which spreads its stores over the banks; the other buffers, and always the final one, are
// unpadded. Buffer capacity: fft_buf_len(L, C) values.
constexpr int FFT_PAD = 4;
__host__ __device__ constexpr int fft_buf_len(int L, int C) { return L * C + ((L * C) >> FFT_PAD) + 1; }

// w_P^(j k) = exp(-2 pi i j k / P) of the direct DFTs (P = 23, 29, 31), row k: read uniformly by a warp, from constant memory
template <int P>
struct DirectCoef {
  float2 w[P * P] = {};
  constexpr DirectCoef() {
    for (int k = 0; k < P; k++)
      for (int j = 0; j < P; j++) {
        double c = 0, s = 0;
        ct_sincos((j * k) % P, P, c, s);
        w[k * P + j].x = (float)c;
        w[k * P + j].y = (float)(-s);
      }
  }
};
__constant__ DirectCoef<23> c_direct23{};
__constant__ DirectCoef<29> c_direct29{};
__constant__ DirectCoef<31> c_direct31{};
template <int P>
__device__ __forceinline__ const float2* direct_coef() {
  if constexpr (P == 23) return c_direct23.w;
  else if constexpr (P == 29) return c_direct29.w;
  else return c_direct31.w;
}

// Shared memory by 32-bit addresses: the stages are functions of their own, and through a generic pointer each of their
// accesses would cost 64-bit address arithmetic and the generic path.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float2 lds2(unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts2(unsigned a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}

// threads that share a butterfly's outputs: the direct sums' (a line of 841 = 29 29 has 29 butterflies per stage)
__host__ __device__ constexpr int butterfly_share(int P) { return P >= 23 ? 4 : 1; }
// The butterfly of radix P on inputs in(j), j < P, with outputs through emit(k, value) (which applies the inter-stage
// twiddle); part: which of butterfly_share(P) parts of the outputs.
template <int P, class C2, class In, class Emit>
__device__ __forceinline__ void butterfly(In in, Emit emit, bool inv, int part = 0) {
  if constexpr (P == 2) {
    C2 a0 = in(0), a1 = in(1);
    emit(0, cadd(a0, a1));
    emit(1, csub(a0, a1));
  } else if constexpr (P == 4) {
    C2 a0 = in(0), a1 = in(1), a2 = in(2), a3 = in(3);
    C2 t0 = cadd(a0, a2), t1 = csub(a0, a2);
    C2 t2 = cadd(a1, a3), t3 = rot(csub(a1, a3), inv);
    emit(0, cadd(t0, t2));
    emit(2, csub(t0, t2));
    emit(1, cadd(t1, t3));
    emit(3, csub(t1, t3));
  } else if constexpr (P == 8) {
    C2 v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = in(j);
    C2 e[4], d[4];
    {
      C2 t0 = cadd(v[0], v[4]), t1 = csub(v[0], v[4]);
      C2 t2 = cadd(v[2], v[6]), t3 = rot(csub(v[2], v[6]), inv);
      e[0] = cadd(t0, t2); e[2] = csub(t0, t2); e[1] = cadd(t1, t3); e[3] = csub(t1, t3);
    }
    {
      C2 t0 = cadd(v[1], v[5]), t1 = csub(v[1], v[5]);
      C2 t2 = cadd(v[3], v[7]), t3 = rot(csub(v[3], v[7]), inv);
      d[0] = cadd(t0, t2); d[2] = csub(t0, t2); d[1] = cadd(t1, t3); d[3] = csub(t1, t3);
    }
    // w8^k, k = 1..3: (h, -h), (0, -1), (-h, -h) forward; conjugates inverse (h = cos(pi / 4))
    constexpr float h = 0.70710678118654752440f;
    const float sg = inv ? 1.f : -1.f;
    C2 t1 = mkc<C2>(h * (d[1].x - sg * d[1].y), h * (d[1].y + sg * d[1].x));
    C2 t2 = mkc<C2>(-sg * d[2].y, sg * d[2].x);
    C2 t3 = mkc<C2>(h * (-d[3].x - sg * d[3].y), h * (-d[3].y + sg * d[3].x));
    emit(0, cadd(e[0], d[0]));
    emit(4, csub(e[0], d[0]));
    emit(1, cadd(e[1], t1));
    emit(5, csub(e[1], t1));
    emit(2, cadd(e[2], t2));
    emit(6, csub(e[2], t2));
    emit(3, cadd(e[3], t3));
    emit(7, csub(e[3], t3));
  } else if constexpr (P == 3 || P == 5 || P == 7 || P == 11 || P == 13 || P == 17 || P == 19) {
    odd_butterfly<P, C2>(in, inv, emit);
  } else {  // the direct sum, inputs in registers, two outputs at a time; the inverse as conj(forward(conj))
    static_assert(P == 23 || P == 29 || P == 31, "a radix with a butterfly");
    C2 v[P];
#pragma unroll
    for (int j = 0; j < P; j++) {
      v[j] = in(j);
      if (inv) v[j].y = -v[j].y;
    }
    const float2* W = direct_coef<P>();
#pragma unroll 1
    for (int k = 2 * part; k < P; k += 2 * butterfly_share(P)) {
      const float2 *w0 = W + k * P, *w1 = W + (k + 1 < P ? k + 1 : k) * P;
      C2 a = v[0], b = v[0];
#pragma unroll
      for (int j = 1; j < P; j++) {
        const float2 p = w0[j], q = w1[j];
        a.x = fmaf(v[j].x, p.x, fmaf(-v[j].y, p.y, a.x));
        a.y = fmaf(v[j].x, p.y, fmaf(v[j].y, p.x, a.y));
        b.x = fmaf(v[j].x, q.x, fmaf(-v[j].y, q.y, b.x));
        b.y = fmaf(v[j].x, q.y, fmaf(v[j].y, q.x, b.y));
      }
      if (inv) {
        a.y = -a.y;
        b.y = -b.y;
      }
      emit(k, a);
      if (k + 1 < P) emit(k + 1, b);
    }
  }
}

// One Stockham stage of radix P from buffer A to buffer B; C interleaved lines of length L, C = 1 << LC. q of a butterfly
// comes from a multiplication by a precomputed reciprocal (magic = ceil(2^32 / s), exact for the sizes here). Radices 2,
// 4, 8 have hand-written butterflies, 3 ... 19 the symmetric odd form, 23, 29 and 31 the direct sum (its inputs in
// registers, its coefficients in constant memory and four threads to a butterfly: rows of 841 = 29 29 take 0.42 ms per
// launch of the row pass at 777 x 1500, 1.25 ms with the inputs read from shared memory for every output). Each radix is its own non-inlined function, so that the registers of one radix's
// butterfly do not add to another's. Butterfly b reads elements b + j istep (b = bi C + l with bi = q s + r). ISH, OSH:
// A, B in the padded layout (only a stage of an even radix with s C < 32 writes it: an odd radix's outputs fall on
// distinct banks as they are). IN, OUT: what the first stage does to its inputs and the last to its outputs.
enum FftIn { IN_PLAIN, IN_CHIRP, IN_MUL, IN_MULCHIRP };
enum FftOut { OUT_PLAIN, OUT_FILT, OUT_CHIRP };
// the operands of IN and OUT: Bluestein's chirp w (values i < L; a line's elements beyond L are 0) and filter f, the
// conjugations of its inverse form, and the responses' factor (hx + omx omy) exb ey by of a column pair (row table yt of
// (omy, ey by))
struct StageEx {
  int L;
  bool conj;
  const float2* w;
  const float2* f;
  const float2* yt;
  float hx, omx, exb;
};

template <int IN>
__device__ __forceinline__ float2 stage_in(unsigned a, int i, int lc, const StageEx& ex) {
  if constexpr (IN == IN_PLAIN) return lds2(a);
  const int e = i >> lc;
  float2 v = make_float2(0.f, 0.f);
  if (IN == IN_MUL || e < ex.L) {
    v = lds2(a);
    if constexpr (IN == IN_MUL || IN == IN_MULCHIRP) {  // the product rounded by itself (no contraction)
      const float2 t = __ldg(ex.yt + e);
      const float G = fmaf(ex.hx, t.x, ex.omx) * ex.exb * t.y;
      v = make_float2(__fmul_rn(v.x, G), __fmul_rn(v.y, G));
    }
    if constexpr (IN == IN_CHIRP || IN == IN_MULCHIRP) {
      if (ex.conj) v.y = -v.y;
      v = cmul(v, __ldg(ex.w + e));
    }
  }
  return v;
}

template <int P, int LC, int IN, int OUT, bool ISH, bool OSH>
__device__ __noinline__ void stage_loop(unsigned A, unsigned B, int s, int m, unsigned magic,
                                        const float2* __restrict__ stw, bool inv, StageEx ex) {
  constexpr int C = 1 << LC;
  const int LP = s * m;  // L / P
  const int nb = LP << LC, istep = nb, ostep = s << LC;
  // a shared butterfly's parts lie whole warps apart (a warp reads the coefficients uniformly)
  constexpr int SH = butterfly_share(P);
  const int nbw = SH > 1 ? (nb + 31) & ~31 : nb;
  for (int t = threadIdx.x; t < nbw * SH; t += blockDim.x) {
    const int part = SH > 1 ? t / nbw : 0, b = t - part * nbw, l = b & (C - 1), bi = b >> LC;
    if (SH > 1 && b >= nb) continue;
    const int q = s == 1 ? bi : (m == 1 ? 0 : (int)__umulhi((unsigned)bi, magic));
    const int ob = ((bi + (P - 1) * q * s) << LC) + l;
    auto in = [&](int j) {
      const int i = b + j * istep;
      return stage_in<IN>(A + 8u * (unsigned)(ISH ? i + (i >> FFT_PAD) : i), i, LC, ex);
    };
    auto emit = [&](int k, float2 val) {
      if (OUT == OUT_PLAIN && k > 0 && q > 0) {
        val = cmul(val, __ldg(stw + (k - 1) * m + q));
      }
      const int o = ob + k * ostep;
      if constexpr (OUT == OUT_FILT) val = cmul(val, __ldg(ex.f + (o >> LC)));
      if constexpr (OUT == OUT_CHIRP) {
        if ((o >> LC) >= ex.L) return;
        val = cmul(val, __ldg(ex.w + (o >> LC)));
        if (ex.conj) val.y = -val.y;
      }
      sts2(B + 8u * (unsigned)(OSH ? o + (o >> FFT_PAD) : o), val);
    };
    butterfly<P, float2>(in, emit, inv, part);
  }
}

// The same stage with every size known at compile time (radix P, stride S, length L, lines C, layout shifts):
// the quotients, strides and padded offsets fold into constants. IN, OUT: as in stage_loop. stw: the stage's twiddles of
// the transform's direction.
template <int P, int S, int L, int C, int ISH, int OSH, int IN, int OUT>
__device__ __noinline__ void stage_fixed(unsigned A, unsigned B, const float2* __restrict__ stw, bool inv, StageEx ex) {
  constexpr int M = L / (P * S), NB = (L / P) * C, ISTEP = S * M * C, OSTEP = S * C, LC = C == 2 ? 1 : 0;
  static_assert(IN == IN_PLAIN || ISTEP % C == 0, "an element's column is the thread's");
  for (int b = threadIdx.x; b < NB; b += blockDim.x) {
    const int l = b % C, bi = b / C;
    const int q = bi / S, r = bi - q * S;
    const int ob = (r + S * P * q) * C + l;
    auto in = [&](int j) {
      const int i = b + j * ISTEP;
      if constexpr (ISH < 31) return stage_in<IN>(A + 8u * (unsigned)(i + (i >> ISH)), i, LC, ex);
      else return stage_in<IN>(A + 8u * (unsigned)i, i, LC, ex);
    };
    auto emit = [&](int k, float2 val) {
      if (OUT == OUT_PLAIN && M > 1 && k > 0 && q > 0) val = cmul(val, __ldg(stw + (k - 1) * M + q));
      const int o = ob + k * OSTEP;
      if constexpr (OUT == OUT_FILT) val = cmul(val, __ldg(ex.f + o / C));
      if constexpr (OUT == OUT_CHIRP) {
        if (o / C >= ex.L) return;
        val = cmul(val, __ldg(ex.w + o / C));
        if (ex.conj) val.y = -val.y;
      }
      if constexpr (OSH < 31) sts2(B + 8u * (unsigned)(o + (o >> OSH)), val);
      else sts2(B + 8u * (unsigned)o, val);
    };
    butterfly<P, float2>(in, emit, inv);
  }
}

// compile-time plan: the factorisation of fft_make_plan (8s, 4s, 2s, then odd primes up to 31)
struct CPlan {
  int nst = 0, nstw = 0;
  int p[FFT_MAXST] = {}, s[FFT_MAXST] = {}, so[FFT_MAXST] = {};  // so, nstw: the stages' twiddles as in FftPlan
};
constexpr CPlan cplan(int L) {
  CPlan c{};
  int m = L, f[FFT_MAXST] = {}, n = 0;
  while (m % 8 == 0) { f[n++] = 8; m /= 8; }
  while (m % 4 == 0) { f[n++] = 4; m /= 4; }
  while (m % 2 == 0) { f[n++] = 2; m /= 2; }
  const int primes[10] = {3, 5, 7, 11, 13, 17, 19, 23, 29, 31};
  for (int i = 0; i < 10; i++)
    while (m % primes[i] == 0) { f[n++] = primes[i]; m /= primes[i]; }
  int st = 1;
  for (int i = 0; i < n; i++) {
    c.p[i] = f[i];
    c.s[i] = st;
    st *= f[i];
    c.so[i] = c.nstw;
    c.nstw += (f[i] - 1) * (L / st);
  }
  c.nst = n;
  return c;
}

// whether stage st of a fixed plan writes the padded layout (as fft_stage decides for the runtime plans)
constexpr bool stage_pads(const CPlan& P, int st, int C) { return P.p[st] % 2 == 0 && st + 1 < P.nst && P.s[st] * C < 32; }

// the fixed plan of length L from stage ST on: stage 0 reads `first` through IN, the last stage writes through OUT; the
// stages write b, a, b, ... (ST = 0: first may be a), the last one dst where that is not null (neither buffer); returns
// the buffer holding the result
template <int L, int C, int ST, int IN, int OUT>
__device__ __forceinline__ float2* fft_run_fixed(const float2* first, float2* a, float2* b, float2* dst, const FftPlan& pl,
                                                 bool inv, const StageEx& ex) {
  constexpr CPlan P = cplan(L);
  if constexpr (ST == P.nst) {
    return a;
  } else {
    constexpr int OSH = stage_pads(P, ST, C) ? FFT_PAD : 31;
    constexpr int ISH = ST > 0 && stage_pads(P, ST > 0 ? ST - 1 : 0, C) ? FFT_PAD : 31;
    float2* to = ST + 1 == P.nst && dst ? dst : b;
    stage_fixed<P.p[ST], P.s[ST], L, C, ISH, OSH, ST == 0 ? IN : (int)IN_PLAIN, ST + 1 == P.nst ? OUT : (int)OUT_PLAIN>(
        smem_addr(first), smem_addr(to), pl.stw + P.so[ST] + (inv ? P.nstw : 0), inv, ex);
    __syncthreads();
    return fft_run_fixed<L, C, ST + 1, IN, OUT>(b, to, a, dst, pl, inv, ex);
  }
}

// stage st of the plan from A (padded: ish) to B; returns whether B is padded
template <int LC, int IN, int OUT>
__device__ __forceinline__ bool fft_stage(const float2* A, float2* B, const FftPlan& pl, int st, int SL, bool inv, bool ish,
                                          const StageEx& ex) {
  const int P = pl.p[st], s = pl.s[st], m = SL / (P * s);
  const bool osh = P % 2 == 0 && st + 1 < pl.nst && (s << LC) < 32;
  auto go = [&](auto pc) {
    constexpr int PP = decltype(pc)::value;
    constexpr bool EVEN = PP == 2 || PP == 4 || PP == 8;
    auto call = [&](auto ic, auto oc) {
      constexpr bool IS = decltype(ic)::value && IN == IN_PLAIN, OS = decltype(oc)::value && EVEN && OUT == OUT_PLAIN;
      stage_loop<PP, LC, IN, OUT, IS, OS>(smem_addr(A), smem_addr(B), s, m, pl.magic[st], pl.stw + pl.so[st] + (inv ? pl.nstw : 0), inv, ex);
    };
    if (ish) {
      if (EVEN && osh) call(std::true_type{}, std::true_type{});
      else call(std::true_type{}, std::false_type{});
    } else {
      if (EVEN && osh) call(std::false_type{}, std::true_type{});
      else call(std::false_type{}, std::false_type{});
    }
  };
  using std::integral_constant;
  switch (P) {
    case 2: go(integral_constant<int, 2>{}); break;
    case 3: go(integral_constant<int, 3>{}); break;
    case 4: go(integral_constant<int, 4>{}); break;
    case 5: go(integral_constant<int, 5>{}); break;
    case 7: go(integral_constant<int, 7>{}); break;
    case 8: go(integral_constant<int, 8>{}); break;
    case 11: go(integral_constant<int, 11>{}); break;
    case 13: go(integral_constant<int, 13>{}); break;
    case 17: go(integral_constant<int, 17>{}); break;
    case 19: go(integral_constant<int, 19>{}); break;
    case 23: go(integral_constant<int, 23>{}); break;
    case 29: go(integral_constant<int, 29>{}); break;
    default: go(integral_constant<int, 31>{}); break;
  }
  __syncthreads();
  return osh;
}

// the plan's stages on their length SL (L, or Bluestein's M): the first reads `first` (a or neither buffer) through IN and
// writes b, the next ones a, b, ... in turn, the last writes through OUT (first and result unpadded). The result goes to
// dst, which is neither a nor b (it may be `first`: only the first of two or more stages reads that), or for a null dst to
// the buffer that the last stage does not read; returned is where it is.
template <int LC, int IN, int OUT>
__device__ __forceinline__ float2* fft_stages(const float2* first, float2* a, float2* b, float2* dst, const FftPlan& pl,
                                              int SL, bool inv, const StageEx& ex) {
  if (pl.nst == 1) {  // a line of one radix (the testing entry's: a padded line has two stages at least)
    fft_stage<LC, IN, OUT_PLAIN>(first, b, pl, 0, SL, inv, false, ex);
    return b;
  }
  bool ish = fft_stage<LC, IN, OUT_PLAIN>(first, b, pl, 0, SL, inv, false, ex);
  float2 *x = b, *y = a;
  for (int st = 1; st + 1 < pl.nst; st++) {
    ish = fft_stage<LC, IN_PLAIN, OUT_PLAIN>(x, y, pl, st, SL, inv, ish, ex);
    float2* t = x;
    x = y;
    y = t;
  }
  float2* to = dst ? dst : y;
  fft_stage<LC, IN_PLAIN, OUT>(x, to, pl, pl.nst - 1, SL, inv, ish, ex);
  return to;
}
// A line of one stage has no place for OUT and a dst. The lengths that have one are the radices, at most 31; a padded line
// and a Bluestein inner length (at least 2 * 37 - 1) are longer.
static_assert(2 * PAD + 1 > 31, "a padded line has two stages at least");

// The 16 inner lengths that fft_work_length gives most of the 1316 lengths from 160 to 2048 with a prime factor above 31
// (the 16th serves 26 of them, all together 69 %; a further length costs 13 s of compile time and serves under 2 %).
#define FFT_INNER_LENGTHS(X) \
  X(1352) X(1463) X(1573) X(1672) X(1859) X(1976) X(2197) X(2431)                                  \
  X(2527) X(2717) X(2873) X(3211) X(3328) X(3584) X(3757) X(4096)

// Bluestein with the inner length FM fixed at compile time (L still read at run time): fft_bluestein's contract
template <int FM, int LC, int IN>
__device__ __noinline__ float2* fft_bluestein_fixed(const float2* first, float2* a, float2* b, float2* dst,
                                                    const FftPlan& pl, bool inv, StageEx ex) {
  constexpr int C = 1 << LC, CHIRP = IN == IN_MUL ? (int)IN_MULCHIRP : (int)IN_CHIRP;
  float2* r = fft_run_fixed<FM, C, 0, CHIRP, OUT_FILT>(first, a, b, nullptr, pl, false, ex);
  return fft_run_fixed<FM, C, 0, IN_PLAIN, OUT_CHIRP>(r, r, r == a ? b : a, dst, pl, true, ex);
}

// Bluestein (the plan's M > 0): X_k = w_k sum_n (x_n w_n) conj(w_{k - n}), w_n = exp(-i pi n^2 / L), the convolution
// cyclic over M >= 2L - 1 by two length-M transforms; the inverse transform as conj(forward(conj(x))). The products by
// the chirp and the filter are made as the transforms' first stages load and their last stages store. `first` holds the
// line's L values (x C); a and b fft_buf_len(M, C) values each (first may be a); the result goes to dst (its L values;
// may be `first`), or for a null dst to a or b. FM > 0: M is FM. The inner lengths that the most padded sizes take
// (FFT_INNER_LENGTHS) have stages of their own, compiled for the default factor order: the strides, offsets and the
// quotient by them are constants, where the runtime stages, bound by issued instructions, spend a third of them there
// (response row pass: M = 2873, 1367 x 911, 444 -> 352 us; 1859, 853 x 1475, 505 -> 346 us; 4096, 1900 x 1977,
// 1267 -> 980 us; the same values). Other inner lengths, and a plan in another factor order, run the runtime stages.
template <int LC, int IN, int FM = 0>
__device__ __forceinline__ float2* fft_bluestein(const float2* first, float2* a, float2* b, float2* dst, const FftPlan& pl,
                                                 bool inv, StageEx ex) {
  ex.L = pl.L;
  ex.conj = inv;
  ex.w = pl.chirp;
  ex.f = pl.filt;
  if constexpr (FM > 0) {
    return fft_bluestein_fixed<FM, LC, IN>(first, a, b, dst, pl, inv, ex);
  } else {
    switch (pl.inner) {
#define INNER_CASE(M) case M: return fft_bluestein_fixed<M, LC, IN>(first, a, b, dst, pl, inv, ex);
      FFT_INNER_LENGTHS(INNER_CASE)
#undef INNER_CASE
      default: break;
    }
    float2* r = fft_stages<LC, IN == IN_MUL ? IN_MULCHIRP : IN_CHIRP, OUT_FILT>(first, a, b, nullptr, pl, pl.M, false, ex);
    return fft_stages<LC, IN_PLAIN, OUT_CHIRP>(r, r, r == a ? b : a, dst, pl, pl.M, true, ex);
  }
}

// a runtime plan's transform of the line(s) in `first` (L values x C, not kept) with two scratch buffers of
// fft_buf_len(work length, C); the result goes to dst, which is neither scratch buffer
template <int FIXL, int LC>
__device__ __forceinline__ void fft_run_to(const float2* first, float2* a, float2* b, float2* dst, const FftPlan& pl, bool inv) {
  if constexpr (FIXL == -1) fft_bluestein<LC, IN_PLAIN>(first, a, b, dst, pl, inv, StageEx{});
  else fft_stages<LC, IN_PLAIN, OUT_PLAIN>(first, a, b, dst, pl, pl.L, inv, StageEx{});
}

// runs the plan on buf (tmp: scratch of the same capacity, fft_buf_len(fft_work_len(pl), C)); buf holds the input
// unpadded and the returned buffer the result unpadded. FIXL > 0: the length is FIXL and the plan is fixed at
// compile time; FIXL = 0: a runtime plan transformed directly; FIXL = -1: a runtime Bluestein plan (kernels are
// instantiated per FIXL, so that each carries only its own path's code and registers).
template <int FIXL, int C, class C2>
__device__ C2* fft_run(C2* buf, C2* tmp, const FftPlan& pl, bool inv) {
  static_assert(C == 1 || C == 2, "C: one line or a pair");
  static_assert(std::is_same<C2, float2>::value, "float32 transforms");
  constexpr int LC = C == 2 ? 1 : 0;
  if constexpr (FIXL > 0) {
    return fft_run_fixed<FIXL, C, 0, IN_PLAIN, OUT_PLAIN>(buf, buf, tmp, nullptr, pl, inv, StageEx{});
  } else if constexpr (FIXL == -1) {  // the kernels' instantiation for Bluestein plans (pl.M > 0)
    return fft_bluestein<LC, IN_PLAIN>(buf, buf, tmp, nullptr, pl, inv, StageEx{});
  } else if constexpr (FIXL < -1) {  // Bluestein with the inner length -FIXL fixed at compile time
    return fft_bluestein<LC, IN_PLAIN, -FIXL>(buf, buf, tmp, nullptr, pl, inv, StageEx{});
  } else {
    return fft_stages<LC, IN_PLAIN, OUT_PLAIN>(buf, buf, tmp, nullptr, pl, pl.L, inv, StageEx{});
  }
}

// z^e, 0 <= e < 64, of the B-spline pole z = sqrt(3) - 2 (interp.py:9): the product of its binary powers z^(2^b),
// formed in float64 at compile time and rounded once
constexpr double BZ1 = -0.26794919243112270, BZ2 = BZ1 * BZ1, BZ4 = BZ2 * BZ2, BZ8 = BZ4 * BZ4, BZ16 = BZ8 * BZ8,
                 BZ32 = BZ16 * BZ16;
__device__ __forceinline__ float zpow(int e) {
  float r = (e & 1) ? (float)BZ1 : 1.f;
  r *= (e & 2) ? (float)BZ2 : 1.f;
  r *= (e & 4) ? (float)BZ4 : 1.f;
  r *= (e & 8) ? (float)BZ8 : 1.f;
  r *= (e & 16) ? (float)BZ16 : 1.f;
  r *= (e & 32) ? (float)BZ32 : 1.f;
  return r;
}

// Cubic B-spline prefilter (interp.py:13-27, without the factor 6, which the caller folds into its scale) of C
// interleaved complex lines of length n in buf, given the lines already divided by 4 + 2 cos w on the periodic
// grid (the response multiply folds that factor into the filter). Per axis the recursion's transfer function is
// -z / (1 - 2 z cos w + z^2) = 1 / (4 + 2 cos w), so the periodic division is the recursion on the periodic
// extension; the reference's recursion on the line (causal start sum_{k < 21} z^k x[k], anticausal start
// z / (z^2 - 1) (y[n-1] + z y[n-2])) differs from it by two closed-form edge terms:
//   c[i] = c_per[i] - D0 z^(i+1) / (1 - z^2) + E z^(n-1-i),
//   D0 = y[0] - y_per[0] = sum_{k < 21} z^k x[k] - sum_{k >= 0} z^k x[-k],  E = c[n-1] - c_per[n-1],
// with x recovered locally as x[i] = c_per[i-1] + 4 c_per[i] + c_per[i+1] (circular) and the sums cut at
// z^32 < 1e-18 (lines here are at least 65 long, so the terms of the two ends never meet). scratch: 2 C float4.
template <int C>
__device__ void bspline_edge_consts(float2* buf, int n, float4* scratch) {
  const float z = (float)BZ1;
  const float g = (float)(BZ1 / (BZ2 - 1.0));
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  auto c = [&](int i, int l) { return buf[(i < 0 ? i + n : (i >= n ? i - n : i)) * C + l]; };
  auto xr = [&](int i, int l) {
    const float2 a = c(i - 1, l), b = c(i, l), d = c(i + 1, l);
    return make_float2(fmaf(4.f, b.x, a.x + d.x), fmaf(4.f, b.y, a.y + d.y));
  };
  for (int l = wid; l < C; l += (int)(blockDim.x >> 5)) {  // a warp per line: its two edge constants, lane k
    const int k = lane;                                       // taking the terms of z^k
    const float zk = zpow(k);
    const int hz = min(n, HORIZON);
    float2 d0 = make_float2(0.f, 0.f);
    if (k < hz) {
      const float2 v = xr(k, l);
      d0 = make_float2(zk * v.x, zk * v.y);
    }
    const float2 w = xr(k == 0 ? 0 : n - k, l);
    d0.x = fmaf(-zk, w.x, d0.x);
    d0.y = fmaf(-zk, w.y, d0.y);
    const float2 ya = xr(n - 1 - k, l), yb = xr(n - 2 - k, l);
    float ax = zk * ya.x, ay = zk * ya.y, bx = zk * yb.x, by = zk * yb.y;
    for (int o = 16; o; o >>= 1) {
      d0.x += __shfl_xor_sync(0xffffffffu, d0.x, o);
      d0.y += __shfl_xor_sync(0xffffffffu, d0.y, o);
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
      bx += __shfl_xor_sync(0xffffffffu, bx, o);
      by += __shfl_xor_sync(0xffffffffu, by, o);
    }
    if (lane == 0) {
      const float2 cl = c(n - 1, l);
      scratch[l] = make_float4(d0.x, d0.y, g * fmaf(z, bx, ax) - cl.x, g * fmaf(z, by, ay) - cl.y);
    }
  }
  __syncthreads();
}

// value v of row j of a line of length n with the edge terms of its constants k added (the first and last 32 rows)
__device__ __forceinline__ float2 bspline_edge_fix(float2 v, int j, int n, float4 k) {
  const float q = (float)(1.0 / (1.0 - BZ2));
  if (j < 32) {
    const float zp = zpow(j + 1);  // z^(i+1), i = j
    v.x = fmaf(-k.x * q, zp, v.x);
    v.y = fmaf(-k.y * q, zp, v.y);
  } else if (j >= n - 32) {
    const float zp = zpow(n - 1 - j);
    v.x = fmaf(k.z, zp, v.x);
    v.y = fmaf(k.w, zp, v.y);
  }
  return v;
}

// the edge constants (bspline_edge_consts) and their terms applied in place
template <int C>
__device__ void bspline_edges(float2* buf, int n, float4* scratch) {
  bspline_edge_consts<C>(buf, n, scratch);
  for (int t = threadIdx.x; t < 64 * C; t += blockDim.x) {
    const int l = t % C, j = t / C;  // j < 32: the start of the line; j >= 32: its end
    const int i = j < 32 ? j : n - 64 + j;
    buf[i * C + l] = bspline_edge_fix(buf[i * C + l], i, n, scratch[l]);
  }
  __syncthreads();
}

// reflect (mirror without repeating the edge, interp.py:38-43) of an index at most one period outside [0, n)
__device__ __forceinline__ int reflect_near(int i, int n) {
  int m = i < 0 ? -i : i;
  if (m >= n) m = 2 * (n - 1) - m;
  if (m < 0 || m >= n) m = (int)mirror_idx(i, n);  // far outside (n tiny): the general rule
  return m;
}

// ---------------------------------------------------------------- kernels
// Every kernel stages its lines in buffers of fft_buf_len(L, C) values (the transforms' padded layouts); the
// prefilter's carries live in the buffer the transform left idle. The kernels are instantiated for FIXL = 0 (any
// supported length, the plan read at run time), FIXL = -1 (Bluestein) and FIXL = each length of fft_fixed_length (the
// padded lengths of 256-, 512-, 768-, 960-, 1024-, 1536- and 2048-wide images: 320, 576, 832, 1024, 1088, 1600,
// 2112 = 8 8 3 11; the plan fixed at compile time), and FIXL = -FFT_FIXED_M (Bluestein with that inner length fixed);
// the launchers pick by the plan.

// the runtime plans' kernels keep to 80 registers (at 128 registers the row pass below took 0.472 ms, at 64 0.60 ms)
constexpr int RT_MINB = 1;
// buffer stride of the kernels that stage several lines: fft_buf_len rounded up to an even count (16-byte aligned)
__host__ __device__ constexpr int fft_buf_stride(int L, int C) { return (fft_buf_len(L, C) + 1) & ~1; }

template <int FIXL>
__global__ void __launch_bounds__(FIXL > 0 || FIXL < -1 ? FFT_TMAX : RT_T, FIXL > 0 || FIXL < -1 ? 2 : RT_MINB) k_fft_rows_fwd_real(const float* __restrict__ img, int W, int H,
                                                                  FftPlan plw, int ph, float2* __restrict__ out) {
  grid_dep_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sm = (float2*)smraw;
  const int pw = FIXL > 0 ? FIXL : plw.L;
  float2* t = sm + fft_buf_len(FIXL > 0 ? FIXL : fft_work_len(plw), 1);
  const int yp = blockIdx.x;
  const int ys = reflect_near(yp - PAD, H);
  const float* row = img + (size_t)ys * W;
  for (int x = threadIdx.x; x < pw; x += blockDim.x) sm[x] = make_float2(__ldg(row + reflect_near(x - PAD, W)), 0.f);
  __syncthreads();
  float2* r = fft_run<FIXL, 1>(sm, t, plw, false);
  float2* o = out + (size_t)yp * pw;
  for (int x = threadIdx.x; x < pw; x += blockDim.x) o[x] = r[x];
}

// The column pass of the responses in two kernels, so that a block holds only two buffers of C columns
// (several blocks per SM instead of one): k_fft_cols_fwd writes the column spectrum S (ph x pw, row-major,
// small enough to stay in L2), then the inverse pass (k_fft_cols_pair, or k_fft_cols_inv_filter where the column
// pair does not fit beside the two buffers) multiplies S by the factors of each plane, inverts along y and stores.
constexpr int COLS_TMAX = 320;  // threads per block of the split column pass

template <int C, int FIXL>
__global__ void __launch_bounds__(FIXL > 0 || FIXL < -1 ? COLS_TMAX : RT_T, FIXL > 0 || FIXL < -1 ? 3 : RT_MINB) k_fft_cols_fwd(const float2* Tin, FftPlan plh, int pw, float2* S) {
  grid_dep_wait();
  constexpr int LC = C == 4 ? 2 : (C == 2 ? 1 : 0);
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* A = (float2*)smraw;
  const int ph = FIXL > 0 ? FIXL : plh.L, n = ph * C;
  float2* B = A + fft_buf_stride(FIXL > 0 ? FIXL : fft_work_len(plh), C);  // 16-byte aligned: the result may be either buffer
  const int x0 = blockIdx.x * C;
  // C = 2 with an even row pitch: each row of the pair is 16 bytes on a 16-byte boundary, copied asynchronously
  const bool rows16 = C == 2 && pw % 2 == 0;
  if (rows16) {
    for (int y = threadIdx.x; y < ph; y += blockDim.x) __pipeline_memcpy_async(A + 2 * y, Tin + (size_t)y * pw + x0, 16);
    __pipeline_commit();
    __pipeline_wait_prior(0);
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      int y = i >> LC, x = x0 + (i & (C - 1));
      A[i] = x < pw ? Tin[(size_t)y * pw + x] : make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  float2* r = fft_run<FIXL, C>(A, B, plh, false);
  if (rows16) {
    for (int y = threadIdx.x; y < ph; y += blockDim.x) *(float4*)(S + (size_t)y * pw + x0) = *(const float4*)(r + 2 * y);
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      int y = i >> LC, x = x0 + (i & (C - 1));
      if (x < pw) S[(size_t)y * pw + x] = r[i];
    }
  }
}

// The inverse column pass with the spectrum of a column pair staged once per block: the block copies its two
// columns of S (ph x 2) into shared memory, then for each of its planes multiplies them by the plane's factor into
// A, inverts along y (A, B) and stores the pair. REFPACK = false: the responses of the k1 filters
// [k1 blockIdx.y, k1 (blockIdx.y + 1)) (x G_k and the B-spline prefilter's periodic factors, inverse,
// the prefilter's edge terms along y) into plane k of U. REFPACK = true: variant v = blockIdx.y of the reference
// pack (S G, S G i fx, S G i fy; factors in float64) of the filters [k0, k1) into plane 3 (k - k0) + v of U.
// A thread's column is fixed (blockDim is even), so the x factors are read once. C = 1: a single column per block, for
// Bluestein plans whose pair would leave an SM's shared memory room for too few blocks.

// threads of the fixed-length column-pair kernel: the responses COLS_TMAX; the reference pack, whose float64 factors
// take more time per element, one per radix-8 butterfly of the two columns (2 x 2112 / 8); the fixed inner length
// (1216 = 8 8 19: 304 radix-8 butterflies, 128 of radix 19) 256 in 3 blocks per SM (960 x 540: 179 -> 173 us against
// COLS_TMAX in 2, the reference pack 232 -> 225 us)
constexpr int PAIR_T_REF = 544, PAIR_T_INNER = 256;
template <bool REFPACK>
constexpr int pair_threads(int fixl) {
  if (fixl > 0) return REFPACK ? PAIR_T_REF : COLS_TMAX;
  return fixl < -1 ? PAIR_T_INNER : RT_T;
}
constexpr int pair_minb(int fixl) { return fixl > 0 ? 2 : (fixl < -1 ? 3 : RT_MINB); }
template <bool REFPACK, int FIXL, int C>
__global__ void __launch_bounds__(pair_threads<REFPACK>(FIXL), pair_minb(FIXL))
    k_fft_cols_pair(const float2* __restrict__ S, FftPlan plh, int pw, GaborTables g, int k0, int k1,
                    float2* __restrict__ U) {
  grid_dep_wait();
  static_assert(C == 2 || FIXL == -1, "one column per block: Bluestein's runtime plans");
  constexpr int LC = C - 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ph = FIXL > 0 ? FIXL : plh.L, n = ph * C, tid = threadIdx.x, nt = blockDim.x;
  float2* raw = (float2*)smraw;
  float2* A = raw + ((n + 1) & ~1);
  float2* B = A + fft_buf_stride(FIXL > 0 ? FIXL : fft_work_len(plh), C);
  const int x0 = blockIdx.x * C;
  const bool rows16 = C == 2 && x0 + 1 < pw && pw % 2 == 0;  // each row of the pair is 16 bytes on a 16-byte boundary
  if (rows16) {
    for (int y = tid; y < ph; y += nt) __pipeline_memcpy_async(raw + 2 * y, S + (size_t)y * pw + x0, 16);
    __pipeline_commit();
    __pipeline_wait_prior(0);
  } else {
    for (int i = tid; i < n; i += nt) {
      const int y = i >> LC, x = x0 + (i & (C - 1));
      raw[i] = x < pw ? S[(size_t)y * pw + x] : make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  const int x = min(x0 + (tid & (C - 1)), pw - 1);
  auto store = [&](const float2* r, int plane) {
    float2* dst = U + (size_t)plane * ph * pw + x0;
    if (rows16) {
      for (int y = tid; y < ph; y += nt) *(float4*)(dst + (size_t)y * pw) = *(const float4*)(r + 2 * y);
    } else {
      for (int i = tid; i < n; i += nt)
        if (x0 + (i & (C - 1)) < pw) dst[(size_t)(i >> LC) * pw + (i & (C - 1))] = r[i];
    }
  };
  // the same with the prefilter's edge terms along y (constants kc of the two columns) added as the rows are stored
  auto store_edges = [&](const float2* r, const float4* kc, int plane) {
    float2* dst = U + (size_t)plane * ph * pw + x0;
    if (rows16) {
      for (int y = tid; y < ph; y += nt) {
        const float4 v = *(const float4*)(r + 2 * y);
        const float2 a = bspline_edge_fix(make_float2(v.x, v.y), y, ph, kc[0]);
        const float2 b = bspline_edge_fix(make_float2(v.z, v.w), y, ph, kc[1]);
        *(float4*)(dst + (size_t)y * pw) = make_float4(a.x, a.y, b.x, b.y);
      }
    } else {
      for (int i = tid; i < n; i += nt)
        if (x0 + (i & (C - 1)) < pw)
          dst[(size_t)(i >> LC) * pw + (i & (C - 1))] = bspline_edge_fix(r[i], i >> LC, ph, kc[i & (C - 1)]);
    }
  };
  if (!REFPACK) {
    const float hx = __ldg(g.hxf + x), omx = __ldg(g.omxf + x), bx = __ldg(g.bxf + x);
    const int kend = min(g.F, (int)(blockIdx.y + 1) * k1);
    for (int k = blockIdx.y * k1; k < kend; k++) {
      // G = (hx + omx omy) ex ey (bx by): the x factors of the thread's column, (omy, ey by) from the row table
      const float exb = __ldg(g.exf + (size_t)k * pw + x) * bx;
      StageEx ex{};
      ex.yt = g.yt2 + (size_t)k * ph;
      ex.hx = hx;
      ex.omx = omx;
      ex.exb = exb;
      float2* r;
      if constexpr (FIXL > 0) r = fft_run_fixed<FIXL, C, 0, IN_MUL, OUT_PLAIN>(raw, A, B, nullptr, plh, true, ex);
      else if constexpr (FIXL < -1) r = fft_bluestein<LC, IN_MUL, -FIXL>(raw, A, B, nullptr, plh, true, ex);
      else if constexpr (FIXL == 0) r = fft_stages<LC, IN_MUL, OUT_PLAIN>(raw, A, B, nullptr, plh, ph, true, ex);
      else r = fft_bluestein<LC, IN_MUL>(raw, A, B, nullptr, plh, true, ex);
      float2* idle = r == A ? B : A;
      bspline_edge_consts<C>(r, ph, (float4*)idle);  // the prefilter's edge terms along y, added by the store
      store_edges(r, (const float4*)idle, k);
      __syncthreads();
    }
  } else {
    const int v = blockIdx.y;
    const double hx = g.hx[x], omx = g.omx[x], fx = g.fx[x];
    for (int k = k0; k < k1; k++) {
      const double ex = g.ex[(size_t)k * pw + x];
      const double* eyk = g.ey + (size_t)k * ph;
      // the row factors omy[y], ey_k[y] (and fy[y]) per element
      auto mul = [&](int i, double omy, double eyv, double fyv) {
        const float2 sv = raw[i];
        const double G = fma(hx, omy, omx) * ex * eyv;
        double re = sv.x * G, im = sv.y * G;
        if (v == 1) { const double t = re; re = -im * fx; im = t * fx; }          // x i fx
        else if (v == 2) { const double t = re; re = -im * fyv; im = t * fyv; }  // x i fy
        A[i] = make_float2((float)re, (float)im);
      };
      if constexpr (FIXL > 0) {
        // the three row factors of UN elements loaded together before their multiplies, so that their latencies
        // overlap (blockDim = PAIR_T_REF)
        constexpr int NT = PAIR_T_REF, NI = (2 * FIXL + NT - 1) / NT, UN = 4;
#pragma unroll
        for (int m0 = 0; m0 < NI; m0 += UN) {
          double oy[UN], ey[UN], fy[UN];
#pragma unroll
          for (int u = 0; u < UN; u++) {
            const int i = threadIdx.x + NT * (m0 + u);
            oy[u] = ey[u] = fy[u] = 0.0;
            if (m0 + u < NI && i < 2 * FIXL) {
              const int y = i >> 1;
              oy[u] = __ldg(g.omy + y);
              ey[u] = __ldg(eyk + y);
              if (v == 2) fy[u] = __ldg(g.fy + y);
            }
          }
#pragma unroll
          for (int u = 0; u < UN; u++) {
            const int i = threadIdx.x + NT * (m0 + u);
            if (m0 + u < NI && i < 2 * FIXL) mul(i, oy[u], ey[u], fy[u]);
          }
        }
      } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
          const int y = i >> LC;
          mul(i, __ldg(g.omy + y), __ldg(eyk + y), v == 2 ? __ldg(g.fy + y) : 0.0);
        }
      }
      __syncthreads();
      float2* r = fft_run<FIXL, C>(A, B, plh, true);
      store(r, 3 * (k - k0) + v);
      __syncthreads();
    }
  }
}

// The same inverse column pass with one block per (C columns, plane) and no staged spectrum: the form for padded
// heights whose column pair does not fit in shared memory beside the two transform buffers.
template <int C, bool REFPACK, int FIXL>
__global__ void __launch_bounds__(RT_T, RT_MINB) k_fft_cols_inv_filter(const float2* __restrict__ S, FftPlan plh, int pw,
                                                                      GaborTables g, int k0, float2* __restrict__ U) {
  constexpr int LC = C == 4 ? 2 : (C == 2 ? 1 : 0);
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* A = (float2*)smraw;
  const int ph = plh.L, n = ph * C;
  float2* B = A + fft_buf_len(fft_work_len(plh), C);
  const int x0 = blockIdx.x * C;
  const int k = REFPACK ? k0 + blockIdx.y / 3 : blockIdx.y, var = REFPACK ? blockIdx.y % 3 : 0;
  const float* exkf = g.exf + (size_t)k * pw;
  const float* eykf = g.eyf + (size_t)k * ph;
  const double* exk = g.ex + (size_t)k * pw;
  const double* eyk = g.ey + (size_t)k * ph;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    int y = i >> LC, xr = x0 + (i & (C - 1)), x = min(xr, pw - 1);
    float2 sv = xr < pw ? S[(size_t)y * pw + x] : make_float2(0.f, 0.f);
    if (!REFPACK) {
      // the Gabor factor and the B-spline prefilter on the periodic grid along both axes
      float G = fmaf(__ldg(g.hxf + x), __ldg(g.omyf + y), __ldg(g.omxf + x)) * (__ldg(exkf + x) * __ldg(eykf + y)) *
                (__ldg(g.bxf + x) * __ldg(g.byf + y));
      A[i] = make_float2(sv.x * G, sv.y * G);
    } else {
      double G = fma(g.hx[x], g.omy[y], g.omx[x]) * exk[x] * eyk[y];
      double re = sv.x * G, im = sv.y * G;
      if (var == 1) { double f = g.fx[x]; double t = re; re = -im * f; im = t * f; }        // x i fx
      else if (var == 2) { double f = g.fy[y]; double t = re; re = -im * f; im = t * f; }   // x i fy
      A[i] = make_float2((float)re, (float)im);
    }
  }
  __syncthreads();
  float2* r = fft_run<FIXL, C>(A, B, plh, true);
  if (!REFPACK) {
    float2* idle = r == A ? B : A;
    bspline_edges<C>(r, ph, (float4*)(((uintptr_t)idle + 15) & ~(uintptr_t)15));  // the prefilter's edge terms along y
  }
  float2* dst = U + (size_t)blockIdx.y * ph * pw;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    int y = i >> LC, x = x0 + (i & (C - 1));
    if (x < pw) dst[(size_t)y * pw + x] = r[i];
  }
}

// Inverse row transforms of the filtered spectra into the responses R, persistent: a block walks the node rows
// blockIdx.x, + gridDim.x, ...; per node row it transforms the row's two lines one after the other, each followed by
// the prefilter's edge terms along x, and stores both at once with the scale 36 / (ph pw).
// R holds the filters in pairs, node-major: pair j = filters 2j and 2j + 1 (the second a copy of filter F - 1 when F
// is odd), filter 2j + c at node (y, x) at R[((j ph + y) pw + x) 2 + c], so that one 16-byte load takes a tap of both
// filters of a pair, and node row (j, y) is one run of pw 16-byte stores.
// Four line buffers: the first line's result waits in one while the second line is transformed in two others, and the
// fourth receives the next row's first line (cp.async) meanwhile; the next row's second line is copied while its
// first line is transformed. (Both lines in one interleaved transform waits longer at the Stockham barriers of its
// 512-thread blocks: 0.377 ms per launch at 2112; one line per block with 8-byte stores 16 bytes apart: 0.36 ms.)
template <int FIXL>
__global__ void __launch_bounds__(FIXL > 0 ? 288 : FFT_TMAX, FIXL > 0 ? 3 : 2)
    k_fft_rows_inv_resp(const float2* __restrict__ U, FftPlan plw, int ph, int F, int nrows, float scale,
                        float2* __restrict__ R) {
  grid_dep_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = FIXL > 0 ? FIXL : plw.L, nb = fft_buf_stride(FIXL > 0 ? FIXL : fft_work_len(plw), 1);
  float2* b0 = (float2*)smraw;
  float2 *x0 = b0, *x1 = b0 + nb, *fa = b0 + 2 * nb, *fb = b0 + 3 * nb;
  // copies line c of node row `row` into dst as one group of asynchronous copies (an empty group past the end)
  auto fetch = [&](int row, int c, float2* dst) {
    if (row < nrows) {
      const int j = row / ph, y = row - j * ph;
      const float2* src = U + ((size_t)min(2 * j + c, F - 1) * ph + y) * L;
      if (L % 2 == 0) {  // 16-byte chunks: the line starts on a 16-byte boundary
        for (int i = threadIdx.x; i < L / 2; i += blockDim.x) __pipeline_memcpy_async(dst + 2 * i, src + 2 * i, 16);
      } else {
        for (int i = threadIdx.x; i < L; i += blockDim.x) __pipeline_memcpy_async(dst + i, src + i, 8);
      }
    }
    __pipeline_commit();
  };
  int row = blockIdx.x;
  fetch(row, 0, x0);
  fetch(row, 1, x1);
  for (; row < nrows; row += gridDim.x) {
    const int nxt = row + gridDim.x;
    __pipeline_wait_prior(1);  // line 0 has landed (line 1 may be in flight)
    __syncthreads();
    float2* r0 = fft_run<FIXL, 1>(x0, fa, plw, true);
    float2* s0 = r0 == x0 ? fa : x0;
    bspline_edge_consts<1>(r0, L, (float4*)s0);  // the edge terms along x, added by the store
    const float4 k0 = *(const float4*)s0;        // s0 is line 1's transform buffer next
    fetch(nxt, 0, fb);         // the next row's line 0 during line 1's transform
    __pipeline_wait_prior(1);  // line 1 has landed
    __syncthreads();
    float2* r1 = fft_run<FIXL, 1>(x1, s0, plw, true);
    float2* s1 = r1 == x1 ? s0 : x1;
    bspline_edge_consts<1>(r1, L, (float4*)s1);
    const float4 k1 = *(const float4*)s1;
    float4* o = (float4*)R + (size_t)row * L;
    for (int x = threadIdx.x; x < L; x += blockDim.x) {
      const float2 a = bspline_edge_fix(r0[x], x, L, k0), b = bspline_edge_fix(r1[x], x, L, k1);
      o[x] = make_float4(a.x * scale, a.y * scale, b.x * scale, b.y * scale);
    }
    __syncthreads();
    // free now: r0, r1 and s1; the next row's line 0 is in fb
    fetch(nxt, 1, s1);
    x0 = fb;
    x1 = s1;
    fa = r0;
    fb = r1;
  }
  __pipeline_wait_prior(0);
}

// The same pass for runtime plans (times of 1367 x 911, rows of 1431 values, Bluestein's M = 2873 = 13 13 17: 0.451 ms per
// launch; 0.838 ms with the four buffers of M, uncoalesced twiddles and separate passes for the chirp and filter products):
// a block takes one node row. The two raw lines keep buffers of L values and receive
// their own results; only the two scratch buffers have the work length (Bluestein's M is about 2 L). More blocks fit per
// SM than with four buffers of M and a prefetch of the next row, and blocks of few threads (rt_threads) leave few
// warps without a butterfly in the stages of large radices. Issue slots (59 %) and barriers bound it.
template <int FIXL>
__global__ void __launch_bounds__(RT_T, RT_MINB) k_fft_rows_inv_resp_rt(const float2* __restrict__ U, FftPlan plw, int ph, int F,
                                                                  float scale, float2* __restrict__ R) {
  grid_dep_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = plw.L, nl = fft_buf_stride(L, 1), nb = fft_buf_stride(fft_work_len(plw), 1), row = blockIdx.x;
  float2 *x0 = (float2*)smraw, *x1 = x0 + nl, *a = x1 + nl, *b = a + nb;
  const int j = row / ph, y = row - j * ph;
  for (int c = 0; c < 2; c++) {
    const float2* src = U + ((size_t)min(2 * j + c, F - 1) * ph + y) * L;
    float2* dst = c ? x1 : x0;
    if (L % 2 == 0) {  // 16-byte chunks: the line starts on a 16-byte boundary
      for (int i = threadIdx.x; i < L / 2; i += blockDim.x) __pipeline_memcpy_async(dst + 2 * i, src + 2 * i, 16);
    } else {
      for (int i = threadIdx.x; i < L; i += blockDim.x) __pipeline_memcpy_async(dst + i, src + i, 8);
    }
    __pipeline_commit();
  }
  float4 k[2];
#pragma unroll 1
  for (int c = 0; c < 2; c++) {
    float2* x = c ? x1 : x0;
    if (c == 0) __pipeline_wait_prior(1);  // line 1 may be in flight
    else __pipeline_wait_prior(0);
    __syncthreads();
    fft_run_to<FIXL, 0>(x, a, b, x, plw, true);
    bspline_edge_consts<1>(x, L, (float4*)a);  // the edge terms along x, added by the store
    k[c] = *(const float4*)a;
    __syncthreads();
  }
  float4* o = (float4*)R + (size_t)row * L;
  for (int x = threadIdx.x; x < L; x += blockDim.x) {
    const float2 p = bspline_edge_fix(x0[x], x, L, k[0]), q = bspline_edge_fix(x1[x], x, L, k[1]);
    o[x] = make_float4(p.x * scale, p.y * scale, q.x * scale, q.y * scale);
  }
}

template <int FIXL>
__global__ void __launch_bounds__(FIXL > 0 || FIXL < -1 ? FFT_TMAX : RT_T, FIXL > 0 || FIXL < -1 ? 2 : RT_MINB) k_fft_rows_inv_ref(const float2* __restrict__ U, FftPlan plw, int ph, int W,
                                                               int H, int k0, int two, float4* __restrict__ ref4,
                                                               float* __restrict__ amp) {
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sm = (float2*)smraw;
  // runtime plans: rows of L values and two scratch buffers of the work length, the results written over the rows (one
  // scratch buffer and a copy of each result where a direct plan's five buffers do not fit: two = 0)
  constexpr bool RT = FIXL == 0 || FIXL == -1;
  const int pw = FIXL > 0 ? FIXL : plw.L, wl = fft_buf_stride(FIXL > 0 ? FIXL : fft_work_len(plw), 1);
  const int nb = RT ? fft_buf_stride(pw, 1) : wl;
  float2* t = sm + 3 * nb;
  const int y = blockIdx.x, kk = blockIdx.y, k = k0 + kk;  // y: row of the W x H crop
  const size_t plane = (size_t)ph * pw;
  // the three rows in three groups of asynchronous copies: rows 1 and 2 land while row 0 is transformed
  for (int v = 0; v < 3; v++) {
    const float2* src = U + (size_t)(3 * kk + v) * plane + (size_t)(y + PAD) * pw;
    if (pw % 2 == 0) {  // 16-byte chunks: the row starts on a 16-byte boundary
      for (int i = threadIdx.x; i < pw / 2; i += blockDim.x) __pipeline_memcpy_async(sm + v * nb + 2 * i, src + 2 * i, 16);
    } else {
      for (int i = threadIdx.x; i < pw; i += blockDim.x) __pipeline_memcpy_async(sm + v * nb + i, src + i, 8);
    }
    __pipeline_commit();
  }
  float2* rr[3];
  for (int v = 0; v < 3; v++) {
    if (v == 0) __pipeline_wait_prior(2);
    else if (v == 1) __pipeline_wait_prior(1);
    else __pipeline_wait_prior(0);
    __syncthreads();
    if (RT && (FIXL == -1 || two)) {
      if constexpr (RT) fft_run_to<FIXL, 0>(sm + v * nb, t, t + wl, sm + v * nb, plw, true);
      rr[v] = sm + v * nb;
      continue;
    }
    if constexpr (FIXL != -1) {
      float2* res = fft_run<FIXL, 1>(sm + v * nb, t, plw, true);
      if (res != sm + v * nb) {
        for (int x = threadIdx.x; x < pw; x += blockDim.x) sm[v * nb + x] = res[x];
        __syncthreads();
      }
      rr[v] = sm + v * nb;
    }
  }
  const double sc = 1.0 / ((double)ph * (double)pw);
  for (int x = threadIdx.x; x < W; x += blockDim.x) {
    int xp = x + PAD;
    float2 a = rr[0][xp], b = rr[1][xp], c = rr[2][xp];
    double rre = a.x * sc, rim = a.y * sc;
    double xre = b.x * sc, xim = b.y * sc, yre = c.x * sc, yim = c.y * sc;
    double a2 = rre * rre + rim * rim + 1e-12;
    // Im(conj(r) rx) / a2 (phaseflow.py:109-110), one reciprocal for both (stored as float32)
    const double ia2 = 1.0 / a2;
    double gx = (rre * xim - rim * xre) * ia2;
    double gy = (rre * yim - rim * yre) * ia2;
    size_t o = (size_t)k * W * H + (size_t)y * W + x;
    ref4[o] = make_float4((float)rre, (float)rim, (float)gx, (float)gy);
    amp[o] = (float)sqrt(a2);
  }
}

template <int FIXL>
__global__ void __launch_bounds__(FIXL > 0 || FIXL < -1 ? FFT_TMAX : RT_T, FIXL > 0 || FIXL < -1 ? 2 : RT_MINB) k_fft_lines(float2* data, FftPlan pl, int inv) {
  extern __shared__ float2 sm[];
  const int L = FIXL > 0 ? FIXL : pl.L;
  float2* row = data + (size_t)blockIdx.x * L;
  for (int x = threadIdx.x; x < L; x += blockDim.x) sm[x] = row[x];
  __syncthreads();
  float2* r = fft_run<FIXL, 1>(sm, sm + fft_buf_len(FIXL > 0 ? FIXL : fft_work_len(pl), 1), pl, inv != 0);
  for (int x = threadIdx.x; x < L; x += blockDim.x) row[x] = r[x];
}

// ---------------------------------------------------------------- launchers
constexpr size_t SMEM_MAX = 227 * 1024;

static void set_smem(const void* fn, size_t bytes) {
  raise_smem_limit(fn, bytes);
}

static size_t fbytes(int L, int C) { return (size_t)fft_buf_len(L, C) * sizeof(float2); }

// shared memory of a transform with the prefilter's edge terms: two buffers, the idle one holding C float4
// from its first 16-byte boundary
static size_t smem_prefilter(int L, int C, int T) {
  (void)T;
  return std::max<size_t>(2 * fbytes(L, C), fbytes(L, C) + 16 + (size_t)C * sizeof(float4));
}
// k_fft_cols_pair: the C columns (C L values) and two buffers of the work length (L, or Bluestein's M) at the even
// stride
static size_t smem_cols(int L, int WL, int C) {
  return ((size_t)C * L + 1 + 2 * (size_t)fft_buf_stride(WL, C)) / 2 * 2 * sizeof(float2);
}
// k_fft_rows_inv_resp: four line buffers at the even stride
static size_t smem_rows_resp(int L) { return 4 * (size_t)fft_buf_stride(L, 1) * sizeof(float2); }

// calls f with std::integral_constant<int, FIXL> for the kernels' instantiation of a plan: a length with a plan fixed
// at compile time, a Bluestein plan whose inner length -FIXL has one (FIXL < -1), the runtime direct plan (0) or the
// runtime Bluestein plan (-1)
template <class Fn>
static void by_plan(const FftPlan& pl, Fn f) {
  using std::integral_constant;
  if (!pl.M) {
    switch (pl.L) {
      case 320: f(integral_constant<int, 320>{}); return;
      case 576: f(integral_constant<int, 576>{}); return;
      case 832: f(integral_constant<int, 832>{}); return;
      case 1024: f(integral_constant<int, 1024>{}); return;
      case 1088: f(integral_constant<int, 1088>{}); return;
      case 1600: f(integral_constant<int, 1600>{}); return;
      case FFT_FIXED_L: f(integral_constant<int, FFT_FIXED_L>{}); return;
      default: break;
    }
  }
  // the Bluestein inner length of 604 = 4 151 (the padded height of 540-row frames: the CLI's 1080p video at scale 2)
  if (pl.M == FFT_FIXED_M) {
    f(integral_constant<int, -FFT_FIXED_M>{});
    return;
  }
  if (pl.M) f(integral_constant<int, -1>{});
  else f(integral_constant<int, 0>{});
}

bool fft_fixed_length(int L) {
  return L == 320 || L == 576 || L == 832 || L == 1024 || L == 1088 || L == 1600 || L == FFT_FIXED_L;
}

// blocks of a kernel resident at once on the device
static int resident_blocks(const void* fn, int threads, size_t smem) {
  int dev = 0, sms = 0, per = 0;
  OFC_CUDA(cudaGetDevice(&dev));
  OFC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  OFC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem));
  return std::max(per, 1) * sms;
}

// blocks of a persistent launch: as many as are resident at once, at most one per unit of work
static int persistent_blocks(const void* fn, int threads, size_t smem, int work) {
  return std::max(1, std::min(work, resident_blocks(fn, threads, smem)));
}

// The filters a block of the responses' column pass takes in turn from its staged column pair: the count whose waves of
// `resident` blocks take the least time, a block's time being its filters plus 0.4 of one for the staging. Few columns
// (small images) spread their filters over the chip, many stage their pair once for several; between them the count
// that fills the last wave best.
static int resp_group(int pairs, int F, int resident) {
  int best = 1;
  double bc = 1e30;
  for (int G = 1; G <= std::min(F, 6); G++) {
    const long blocks = (long)pairs * ((F + G - 1) / G);
    const double c = (double)((blocks + resident - 1) / resident) * (G + 0.4);
    if (c < bc * 0.999) {
      bc = c;
      best = G;
    }
  }
  return best;
}

bool fft_fits(int ph, int pw) {
  try {
    const int wh = fft_work_length(ph), ww = fft_work_length(pw);
    if (wh == 0 || ww == 0) return false;
    int Tc = std::min(fft_threads(wh, 2), COLS_TMAX);
    if (smem_prefilter(wh, 2, Tc) > SMEM_MAX || 2 * (size_t)fft_buf_stride(wh, 2) * sizeof(float2) > SMEM_MAX) return false;
    return 4 * (size_t)fft_buf_stride(ww, 1) * sizeof(float2) <= SMEM_MAX && smem_rows_resp(ww) <= SMEM_MAX;
  } catch (const Error&) {
    return false;
  }
}

// whether a plan runs on the kernels' runtime instantiations (FIXL 0 or -1)
static bool runtime_plan(const FftPlan& pl) { return pl.M ? pl.M != FFT_FIXED_M : !fft_fixed_length(pl.L); }

void launch_fft_rows_fwd_real(const float* img, int W, int H, const FftPlan& plw, int ph, float2* out, cudaStream_t st) {
  size_t sm = 2 * fbytes(fft_work_len(plw), 1);
  int T = runtime_plan(plw) ? rt_threads(plw, 1, sm) : fft_threads(fft_work_len(plw), 1);
  by_plan(plw, [&](auto fl) {
    constexpr int FL = decltype(fl)::value;
    set_smem((const void*)k_fft_rows_fwd_real<FL>, sm);
    OFC_LAUNCH_PDL(k_fft_rows_fwd_real<FL>, ph, T, sm, st, img, W, H, plw, ph, out);
  });
}

static void cols_fwd(float2* T, const FftPlan& plh, int pw, cudaStream_t st) {
  constexpr int C = 2;
  const int wh = fft_work_len(plh);
  size_t sm_f = 2 * (size_t)fft_buf_stride(wh, C) * sizeof(float2);
  int nt = runtime_plan(plh) ? rt_threads(plh, C, sm_f) : std::min(fft_threads(wh, C), COLS_TMAX);
  // in place: a block reads its C columns whole before it writes their spectrum back
  by_plan(plh, [&](auto fl) {
    constexpr int FL = decltype(fl)::value;
    set_smem((const void*)k_fft_cols_fwd<C, FL>, sm_f);
    OFC_LAUNCH_PDL((k_fft_cols_fwd<C, FL>), div_up(pw, C), nt, sm_f, st, T, plh, pw, T);
  });
}

// the inverse column pass of the responses (REFPACK false, planes = filters) or of the reference pack's filters
// [k0, k1) (planes = 3 (k1 - k0))
template <bool REFPACK>
static void cols_inverse(const float2* S, const FftPlan& plh, int pw, const GaborTables& g, int k0, int k1, float2* U,
                         cudaStream_t st) {
  constexpr int C = 2;
  const int ph = plh.L, wh = fft_work_len(plh);
  const bool rt = runtime_plan(plh);
  const size_t sm_p = smem_cols(ph, wh, 2);
  auto launch_cols = [&](auto fl, auto cc, int nt, size_t sm) {
    constexpr int FL = decltype(fl)::value, CC = decltype(cc)::value;
    const void* fn = (const void*)k_fft_cols_pair<REFPACK, FL, CC>;
    set_smem(fn, sm);
    const int cols = (int)div_up(pw, CC);
    if constexpr (REFPACK) {
      OFC_LAUNCH_PDL((k_fft_cols_pair<true, FL, CC>), dim3(cols, 3), nt, sm, st, S, plh, pw, g, k0, k1, U);
    } else {
      const int G = resp_group(cols, g.F, resident_blocks(fn, nt, sm));
      OFC_LAUNCH_PDL((k_fft_cols_pair<false, FL, CC>), dim3(cols, div_up(g.F, G)), nt, sm, st, S, plh, pw, g, 0, G, U);
    }
  };
  // One column per block where the pair's buffers leave room for too few blocks (Bluestein's lengths of large radices
  // above about 2700; the estimate of rt_threads, a column's 8-byte accesses counted 10 %): 911 x 1367 (M = 2873)
  // 0.641 -> 0.510 ms per launch of the responses. Not at M = 4096 (1900 x 1977: 1.73 against 1.94 ms).
  int nt = std::min(fft_threads(wh, C), COLS_TMAX);
  if (rt) {
    double t1 = 1e300, t2 = 1e300;
    const size_t sm1 = smem_cols(ph, wh, 1);
    const int n1 = rt_threads(plh, 1, sm1, &t1);
    nt = rt_threads(plh, C, std::min(sm_p, SMEM_MAX), &t2);
    if (plh.M && sm_p <= SMEM_MAX && 1.1 * t1 < 0.5 * t2) {
      launch_cols(std::integral_constant<int, -1>{}, std::integral_constant<int, 1>{}, n1, sm1);
      return;
    }
  }
  if (sm_p <= SMEM_MAX) {
    if (fft_fixed_length(ph)) nt = pair_threads<REFPACK>(ph);  // the block size the fixed-length kernel assumes
    else if (plh.M == FFT_FIXED_M) nt = std::min(nt, pair_threads<REFPACK>(-FFT_FIXED_M));
    by_plan(plh, [&](auto fl) { launch_cols(fl, std::integral_constant<int, 2>{}, nt, sm_p); });
    return;
  }
  size_t sm_i = REFPACK ? 2 * fbytes(wh, C) : smem_prefilter(wh, C, nt);
  if (sm_i > SMEM_MAX) throw Error(OFC_ERR_WINDOW, "padded height " + std::to_string(ph) + " too large for the column pass");
  dim3 grid(div_up(pw, C), REFPACK ? 3 * (k1 - k0) : g.F);
  auto launch = [&](auto fl) {
    constexpr int FL = decltype(fl)::value;
    set_smem((const void*)k_fft_cols_inv_filter<C, REFPACK, FL>, sm_i);
    OFC_LAUNCH((k_fft_cols_inv_filter<C, REFPACK, FL>), grid, nt, sm_i, st, S, plh, pw, g, k0, U);
  };
  if (plh.M) launch(std::integral_constant<int, -1>{});
  else launch(std::integral_constant<int, 0>{});
}

void launch_fft_cols_filters(float2* T, const FftPlan& plh, int pw, const GaborTables& g, float2* U, cudaStream_t st) {
  cols_fwd(T, plh, pw, st);
  cols_inverse<false>(T, plh, pw, g, 0, g.F, U, st);
}

void launch_fft_rows_inv_resp(const float2* U, const FftPlan& plw, int ph, int F, float2* R, cudaStream_t st) {
  const float scale = (float)(36.0 / ((double)ph * (double)plw.L));
  const int nrows = ((F + 1) / 2) * ph;
  if (runtime_plan(plw)) {
    const size_t sm = (2 * (size_t)fft_buf_stride(plw.L, 1) + 2 * (size_t)fft_buf_stride(fft_work_len(plw), 1)) * sizeof(float2);
    const int T = rt_threads(plw, 1, sm);
    auto launch = [&](auto fl) {
      constexpr int FL = decltype(fl)::value;
      set_smem((const void*)k_fft_rows_inv_resp_rt<FL>, sm);
      OFC_LAUNCH_PDL(k_fft_rows_inv_resp_rt<FL>, nrows, T, sm, st, U, plw, ph, F, scale, R);
    };
    if (plw.M) launch(std::integral_constant<int, -1>{});
    else launch(std::integral_constant<int, 0>{});
    return;
  }
  const int T = fft_threads(fft_work_len(plw), 1);
  const size_t sm = smem_rows_resp(fft_work_len(plw));
  by_plan(plw, [&](auto fl) {
    constexpr int FL = decltype(fl)::value;
    if constexpr (FL > 0 || FL < -1) {
      const void* fn = (const void*)k_fft_rows_inv_resp<FL>;
      set_smem(fn, sm);
      OFC_LAUNCH_PDL(k_fft_rows_inv_resp<FL>, persistent_blocks(fn, T, sm, nrows), T, sm, st, U, plw, ph, F, nrows, scale,
                 R);
    }
  });
}

void launch_fft_cols_fwd(float2* T, const FftPlan& plh, int pw, cudaStream_t st) { cols_fwd(T, plh, pw, st); }

void launch_fft_cols_ref_f32(const float2* S, const FftPlan& plh, int pw, const GaborTables& g, int k0, int k1,
                             float2* U, cudaStream_t st) {
  cols_inverse<true>(S, plh, pw, g, k0, k1, U, st);
}

void launch_fft_rows_inv_ref_f32(const float2* U, const FftPlan& plw, int ph, int k0, int k1, int W, int H,
                                 float4* ref4, float* amp, cudaStream_t st) {
  const bool rt = runtime_plan(plw);
  const size_t wl = fft_buf_stride(fft_work_len(plw), 1);
  size_t sm = 4 * wl * sizeof(float2);
  const size_t sm2 = (3 * (size_t)fft_buf_stride(plw.L, 1) + 2 * wl) * sizeof(float2);
  const bool two = rt && sm2 <= SMEM_MAX;
  if (two) sm = sm2;
  int T = rt ? rt_threads(plw, 1, sm) : fft_threads(fft_work_len(plw), 1);
  dim3 grid(H, k1 - k0);
  by_plan(plw, [&](auto fl) {
    constexpr int FL = decltype(fl)::value;
    set_smem((const void*)k_fft_rows_inv_ref<FL>, sm);
    OFC_LAUNCH(k_fft_rows_inv_ref<FL>, grid, T, sm, st, U, plw, ph, W, H, k0, two ? 1 : 0, ref4, amp);
  });
}

void launch_fft_lines(float2* data, int lines, const FftPlan& pl, bool inverse, cudaStream_t st) {
  size_t sm = 2 * fbytes(fft_work_len(pl), 1);
  int T = runtime_plan(pl) ? rt_threads(pl, 1, sm) : fft_threads(fft_work_len(pl), 1);
  by_plan(pl, [&](auto fl) {
    constexpr int FL = decltype(fl)::value;
    set_smem((const void*)k_fft_lines<FL>, sm);
    OFC_LAUNCH(k_fft_lines<FL>, lines, T, sm, st, data, pl, inverse ? 1 : 0);
  });
}

}  // namespace ofc
