// Batched cubic 3-D DFT with the conventions of the reference's fft3d
// (CalQ/fft3d.h:25-48): forward = FFTW_FORWARD (exp(-2 pi i jk/N)),
// unnormalised; inverse = FFTW_BACKWARD then every element times 1./N^3.
//
// Three passes (axis 2, 1, 0) make the 3-D transform.  A pass loads one N x N
// tile of a cube (N lines of the transform axis) into shared memory, line by
// line, and runs a mixed-radix Stockham FFT on every line: N = r_1 r_2 ... r_m
// with radix-4 and radix-2 stages first (butterflies of additions and +-i
// swaps), then the odd prime factors in ascending order: radix 3 as a
// butterfly, any other odd radix R as one sum of R terms per output against
// the twiddle table exp(sign 2 pi i m/N) (the stage's input twiddle and its
// R-point DFT folded into one table index), so a prime N is the direct DFT.  Stockham's
// self-sorting form ping-pongs between two line buffers and leaves the result
// in natural order.  The per-point cost is sum(r_i) complex operations instead
// of N, e.g. 4 + 2 + 3 against 24 at N = 24.
//
// Three arithmetic types: double2 (FP64), float2 (FP32) and dfc, FP64 data
// in memory with double-float arithmetic in the passes (each part an
// unevaluated hi + lo float pair, edb_df.cuh): GB300 runs native FP64 at a
// small fraction of its FP32 rate, and the FP64 passes of the batch's step
// were bound by it (2.7 ms per pass at 4096 x N = 24).  Double-float keeps
// about 2^-47 relative per operation.
//
// What little FP64 is left bounds a pass, so it is done once: the twiddles come
// with the launch from the host (every block used to evaluate N sines and
// cosines), and a dfc transform splits its input in the first pass, keeps
// (hi, lo) pairs between the passes (the same 16 bytes) and joins them in the
// last.  Transforms, us, before -> now (with N = 16, 24, 32 compiled in): 256 x
// N = 16 185 -> 55 (dfc), 191 -> 115 (FP64), 92 -> 31 (FP32); 2048 x N = 24 3397 ->
// 1280 (dfc).  A dfc pass that splits or joins still runs the FP64 pipe 75% busy.
#include <math.h>

#include <mutex>
#include <type_traits>

#include "edb_df.cuh"
#include "edb_internal.cuh"

namespace edb {

// complex double-float value: re = rh + rl, im = ih + il
struct __align__(16) dfc {
  float rh, rl, ih, il;
};

namespace {
using df::fast_two_sum;
using df::sdf_add;
using df::sdf_mul;
using df::sdf_neg;

__device__ __forceinline__ float2 dsplit(double x) {
  const float h = (float)x;
  return make_float2(h, (float)(x - (double)h));
}
__device__ __forceinline__ dfc mk_dfc(float2 re, float2 im) { return dfc{re.x, re.y, im.x, im.y}; }
__device__ __forceinline__ float2 dre(const dfc &a) { return make_float2(a.rh, a.rl); }
__device__ __forceinline__ float2 dim(const dfc &a) { return make_float2(a.ih, a.il); }
constexpr int FFT_MAX_STAGES = 16;
constexpr int FFT_THREADS = 256;

struct FftPlan {
  int nst;
  int radix[FFT_MAX_STAGES];
};

// 4s, then 2s, then odd prime factors in ascending order.
FftPlan fft_plan(int N) {
  FftPlan p;
  p.nst = 0;
  int n = N;
  while (n % 4 == 0 && p.nst < FFT_MAX_STAGES) {
    p.radix[p.nst++] = 4;
    n /= 4;
  }
  while (n % 2 == 0 && p.nst < FFT_MAX_STAGES) {
    p.radix[p.nst++] = 2;
    n /= 2;
  }
  for (int f = 3; n > 1 && p.nst < FFT_MAX_STAGES; f += 2)
    while (n % f == 0 && p.nst < FFT_MAX_STAGES) {
      p.radix[p.nst++] = f;
      n /= f;
    }
  return p;
}

template <typename R2>
__device__ __forceinline__ R2 c_add(R2 a, R2 b) {
  R2 r;
  r.x = a.x + b.x;
  r.y = a.y + b.y;
  return r;
}
template <typename R2>
__device__ __forceinline__ R2 c_sub(R2 a, R2 b) {
  R2 r;
  r.x = a.x - b.x;
  r.y = a.y - b.y;
  return r;
}
template <typename R2>
__device__ __forceinline__ R2 c_mul(R2 a, R2 w) {
  R2 r;
  r.x = a.x * w.x - a.y * w.y;
  r.y = a.x * w.y + a.y * w.x;
  return r;
}
template <>
__device__ __forceinline__ dfc c_add<dfc>(dfc a, dfc b) {
  return mk_dfc(sdf_add(dre(a), dre(b)), sdf_add(dim(a), dim(b)));
}
template <>
__device__ __forceinline__ dfc c_sub<dfc>(dfc a, dfc b) {
  return mk_dfc(sdf_add(dre(a), sdf_neg(dre(b))), sdf_add(dim(a), sdf_neg(dim(b))));
}
template <>
__device__ __forceinline__ dfc c_mul<dfc>(dfc a, dfc w) {
  return mk_dfc(sdf_add(sdf_mul(dre(a), dre(w)), sdf_neg(sdf_mul(dim(a), dim(w)))),
                sdf_add(sdf_mul(dre(a), dim(w)), sdf_mul(dim(a), dre(w))));
}
// sign i t (sign = +-1): exact
template <typename R2>
__device__ __forceinline__ R2 c_rot(R2 t, int sign) {
  R2 d;
  d.x = -sign * t.y;
  d.y = sign * t.x;
  return d;
}
template <>
__device__ __forceinline__ dfc c_rot<dfc>(dfc t, int sign) {
  return sign > 0 ? dfc{-t.ih, -t.il, t.rh, t.rl} : dfc{t.ih, t.il, -t.rh, -t.rl};
}
// radix-3 parts: t = v0 - s / 2, u = i h d (h real)
template <typename R2>
__device__ __forceinline__ void r3_parts(R2 v0, R2 sm, R2 df, R2 hw, R2 &t, R2 &u) {
  const auto h = hw.y;
  t.x = v0.x - 0.5f * sm.x;
  t.y = v0.y - 0.5f * sm.y;
  u.x = -h * df.y;
  u.y = h * df.x;
}
template <>
__device__ __forceinline__ void r3_parts<dfc>(dfc v0, dfc sm, dfc df, dfc hw, dfc &t, dfc &u) {
  const float2 h = dim(hw);
  // halving is exact in both parts
  t = mk_dfc(sdf_add(dre(v0), make_float2(-0.5f * sm.rh, -0.5f * sm.rl)),
             sdf_add(dim(v0), make_float2(-0.5f * sm.ih, -0.5f * sm.il)));
  u = mk_dfc(sdf_neg(sdf_mul(h, dim(df))), sdf_mul(h, dre(df)));
}
// memory element <-> working value
template <typename R2, typename G>
__device__ __forceinline__ R2 to_work(G g) {
  return g;
}
template <>
__device__ __forceinline__ dfc to_work<dfc, double2>(double2 g) {
  return mk_dfc(dsplit(g.x), dsplit(g.y));
}
// times a real scale (1 or 1/N^3), then to memory
template <typename R2, typename R, typename G>
__device__ __forceinline__ G from_work(R2 x, R scale) {
  x.x *= scale;
  x.y *= scale;
  return x;
}
template <>
__device__ __forceinline__ dfc from_work<dfc, double, dfc>(dfc x, double) {
  return x;  // between passes: no scale
}
template <>
__device__ __forceinline__ double2 from_work<dfc, double, double2>(dfc x, double scale) {
  if (scale != 1.0) {
    const float2 sc = dsplit(scale);
    x = mk_dfc(sdf_mul(dre(x), sc), sdf_mul(dim(x), sc));
  }
  return make_double2((double)x.rh + (double)x.rl, (double)x.ih + (double)x.il);
}
template <typename R2>
R2 make_tw(double c, double s) {
  R2 w;
  w.x = (decltype(w.x))c;
  w.y = (decltype(w.y))s;
  return w;
}
template <>
dfc make_tw<dfc>(double c, double s) {
  const float ch = (float)c, sh = (float)s;
  return dfc{ch, (float)(c - (double)ch), sh, (float)(s - (double)sh)};
}
// exp(2 pi i r / N), 0 <= r < N, from an angle of at most pi / 4: the rounding of
// an angle of up to 2 pi would be several times that of its sine.  FP64 passes'
// relative error, angles in place -> reduced: N = 10 3.7e-16 -> 2.0e-16, 20 4.1e-16 ->
// 2.2e-16, 32 3.7e-16 -> 2.4e-16.
void unit_root(int r, int N, double &c, double &s) {
  int a = 8 * r;  // of 8 N to the circle
  const bool s_neg = a > 4 * N;
  if (s_neg) a = 8 * N - a;
  const bool c_neg = a > 2 * N;
  if (c_neg) a = 4 * N - a;
  const bool swap = a > N;
  if (swap) a = 2 * N - a;
  const double ang = M_PI * a / (4 * N);
  c = swap ? sin(ang) : cos(ang);
  s = swap ? cos(ang) : sin(ang);
  if (c_neg) c = -c;
  if (s_neg) s = -s;
}
// exp(sign 2 pi i r / N), r = 0 .. N - 1, passed to the kernel by value (so a
// launch recorded into a graph carries it).
constexpr int FFT_MAXN = 64;
template <typename R2>
struct FftTw {
  R2 w[FFT_MAXN];
};
template <typename R2>
const FftTw<R2> &fft_tw(int N, int sign) {
  static std::once_flag once[FFT_MAXN + 1][2];
  static FftTw<R2> tab[FFT_MAXN + 1][2];
  const int s = sign > 0;
  FftTw<R2> &t = tab[N][s];
  std::call_once(once[N][s], [&] {
    for (int r = 0; r < FFT_MAXN; ++r) {
      double c, s;
      unit_root(r % N, N, c, s);
      t.w[r] = make_tw<R2>(c, sign * s);
    }
  });
  return t;
}

// One Stockham stage of radix R (2, 3 or 4) on every line of the tile:
// butterfly j of a line reads src[j + i M] (M = N / R), applies the input
// twiddles w^(i tstep), does the R-point DFT and writes dst[expand(j) + q Ns].
template <int R, typename R2>
__device__ __forceinline__ void fft_stage_pow2(int N, int LS, int Ns, int sign, const R2 *src,
                                               R2 *dst, const R2 *tw) {
  const int M = N / R;
  for (int e = threadIdx.x; e < N * M; e += blockDim.x) {
    const int line = e / M, j = e - line * M;
    const R2 *sl = src + (size_t)line * LS;
    R2 *dl = dst + (size_t)line * LS;
    const int k = j % Ns;
    const int tstep = (N / (Ns * R)) * k;
    R2 v[R];
    v[0] = sl[j];
#pragma unroll
    for (int i = 1; i < R; ++i) v[i] = c_mul(sl[j + i * M], tw[(i * tstep) % N]);
    const int d0 = (j / Ns) * Ns * R + k;
    if (R == 2) {
      dl[d0] = c_add(v[0], v[1]);
      dl[d0 + Ns] = c_sub(v[0], v[1]);
    } else if (R == 3) {
      // w3 = exp(sign 2 pi i / 3) = (-1/2, h), h = tw[N / 3].y = sign sqrt(3)/2:
      // o0 = v0 + s, o1,2 = v0 - s/2 +- i h d  (s = v1 + v2, d = v1 - v2)
      const R2 sm = c_add(v[1], v[2]), df = c_sub(v[1], v[2]);
      R2 t, u;
      r3_parts(v[0], sm, df, tw[N / 3], t, u);
      dl[d0] = c_add(v[0], sm);
      dl[d0 + Ns] = c_add(t, u);
      dl[d0 + 2 * Ns] = c_sub(t, u);
    } else {
      // w4 = exp(sign 2 pi i / 4) = sign i; (v1 - v3) w4
      const R2 a = c_add(v[0], v[2]), b = c_sub(v[0], v[2]), c = c_add(v[1], v[3]);
      const R2 d = c_rot(c_sub(v[1], v[3]), sign);
      dl[d0] = c_add(a, c);
      dl[d0 + Ns] = c_add(b, d);
      dl[d0 + 2 * Ns] = c_sub(a, c);
      dl[d0 + 3 * Ns] = c_sub(b, d);
    }
  }
}

// One Stockham stage of any radix R, one output per thread: output q of
// butterfly j is sum_i src[j + i M] w^(i (tstep + q N / R)), i ascending.
template <typename R2, typename R>
__device__ __forceinline__ void fft_stage_direct(int N, int LS, int Rd, int Ns, const R2 *src,
                                                 R2 *dst, const R2 *tw) {
  const int M = N / Rd;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int line = e / N, p = e - line * N;
    const R2 *sl = src + (size_t)line * LS;
    // p = (j / Ns) Ns R + q Ns + k with k = j mod Ns
    const int k = p % Ns, rest = p / Ns;
    const int q = rest % Rd, j = (rest / Rd) * Ns + k;
    const int step = (N / (Ns * Rd)) * k + q * M;
    R2 o;
    if constexpr (std::is_same<R2, dfc>::value) {
      o = dfc{0.f, 0.f, 0.f, 0.f};
      int m = 0;
      for (int i = 0; i < Rd; ++i) {
        o = c_add(o, c_mul(sl[j + i * M], tw[m]));
        m += step;
        if (m >= N) m %= N;
      }
    } else {
      R sr = 0, si = 0;
      int m = 0;
      for (int i = 0; i < Rd; ++i) {
        const R2 x = sl[j + i * M];
        const R2 w = tw[m];
        sr += x.x * w.x - x.y * w.y;
        si += x.x * w.y + x.y * w.x;
        m += step;
        if (m >= N) m %= N;
      }
      o.x = sr;
      o.y = si;
    }
    dst[(size_t)line * LS + p] = o;
  }
}
// The stages of a size known at compile time, in fft_plan's order.
template <int NC, int Ns, typename R2>
__device__ __forceinline__ void fft_stages(int sign, R2 *&src, R2 *&dst, const R2 *tw) {
  if constexpr (Ns < NC) {
    constexpr int rem = NC / Ns, Rd = rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : 3;
    static_assert(rem % Rd == 0, "sizes of factors 2 and 3");
    fft_stage_pow2<Rd>(NC, NC + 1, Ns, sign, src, dst, tw);
    __syncthreads();
    R2 *x = src;
    src = dst;
    dst = x;
    fft_stages<NC, Ns * Rd>(sign, src, dst, tw);
  }
}
}  // namespace

// One pass: the tile's N lines along `axis` of cube blockIdx.y.
//   axis 2: tile = plane i (t); lines are rows (contiguous k), u = j.
//   axis 1: tile = plane i (t); lines are columns (fixed k), along j.
//   axis 0: tile = rows i of fixed j (t); lines are columns (fixed k), along i.
// Shared memory holds the tile twice (line stride N + 1, so that loading
// columns does not hit one bank) and the twiddle table.  in may alias out
// (passes 2 and 3 run in place, element sizes equal): every global read happens
// before the first barrier and every write after the last.
// NC > 0: N known at compile time (the workloads' sizes): the stage loops'
// divisions and remainders by N, N / R and Ns fold away.
template <int NC, typename R2, typename R, typename GI, typename GO>
__global__ void fft_pass_kernel(int n_, int axis, int sign, R scale, FftPlan plan,
                                const __grid_constant__ FftTw<R2> twt, const GI *in, GO *out) {
  extern __shared__ unsigned char smem_raw[];
  const int N = NC > 0 ? NC : n_;
  const int LS = N + 1;
  R2 *buf0 = reinterpret_cast<R2 *>(smem_raw);  // [N][LS]
  R2 *buf1 = buf0 + (size_t)N * LS;              // [N][LS]
  R2 *tw = buf1 + (size_t)N * LS;                // [N]
  const long long NQ = (long long)N * N * N;
  const long long NN = (long long)N * N;
  const int cube = blockIdx.y;
  const int t = blockIdx.x;
  long long base, row_stride;
  if (axis == 0) {
    base = (long long)cube * NQ + (long long)t * N;
    row_stride = NN;
  } else {
    base = (long long)cube * NQ + (long long)t * NN;
    row_stride = N;
  }
  // tile element (u, v): u = row, v = column (contiguous in memory)
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int u = e / N, v = e - u * N;
    const R2 x = to_work<R2, GI>(in[base + (long long)u * row_stride + v]);
    if (axis == 2)
      buf0[(size_t)u * LS + v] = x;
    else
      buf0[(size_t)v * LS + u] = x;
  }
  for (int r = threadIdx.x; r < N; r += blockDim.x) tw[r] = twt.w[r];
  __syncthreads();
  R2 *src = buf0, *dst = buf1;
  if constexpr (NC > 0) fft_stages<NC, 1>(sign, src, dst, tw);
  int Ns = 1;
  for (int s = 0; NC == 0 && s < plan.nst; ++s) {
    const int Rd = plan.radix[s];
    if (Rd == 4)
      fft_stage_pow2<4>(N, LS, Ns, sign, src, dst, tw);
    else if (Rd == 2)
      fft_stage_pow2<2>(N, LS, Ns, sign, src, dst, tw);
    else if (Rd == 3)
      fft_stage_pow2<3>(N, LS, Ns, sign, src, dst, tw);
    else
      fft_stage_direct<R2, R>(N, LS, Rd, Ns, src, dst, tw);
    __syncthreads();
    R2 *x = src;
    src = dst;
    dst = x;
    Ns *= Rd;
  }
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int u = e / N, v = e - u * N;
    const R2 x = (axis == 2) ? src[(size_t)u * LS + v] : src[(size_t)v * LS + u];
    out[base + (long long)u * row_stride + v] = from_work<R2, R, GO>(x, scale);
  }
}

template <int NC, typename R2, typename R, typename GI, typename GO>
static edb_status fft_pass_n(int N, int batch, int axis, int sign, R scale, const FftPlan &plan,
                           const GI *in, GO *out, cudaStream_t st) {
  static_assert(sizeof(GI) == sizeof(GO), "passes run in place");
  auto kern = fft_pass_kernel<NC, R2, R, GI, GO>;
  // once per instantiation, thread-safe (N = 64 in FP64 needs 131 KB)
  static const cudaError_t configured =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (configured != cudaSuccess) return cuda_fail(configured, "cudaFuncSetAttribute(fft_pass)");
  const int threads = N * N < FFT_THREADS ? ((N * N + 31) / 32) * 32 : FFT_THREADS;
  const size_t smem = sizeof(R2) * (2 * (size_t)N * (N + 1) + N);
  kern<<<dim3((unsigned)N, (unsigned)batch), threads, smem, st>>>(N, axis, sign, scale, plan,
                                                                  fft_tw<R2>(N, sign), in, out);
  EDB_LAUNCHED();
  return EDB_OK;
}

template <typename R2, typename R, typename GI, typename GO>
static edb_status fft_pass(int N, int batch, int axis, int sign, R scale, const FftPlan &plan,
                           const GI *in, GO *out, cudaStream_t st) {
  switch (N) {
    case 16: return fft_pass_n<16, R2, R, GI, GO>(N, batch, axis, sign, scale, plan, in, out, st);
    case 24: return fft_pass_n<24, R2, R, GI, GO>(N, batch, axis, sign, scale, plan, in, out, st);
    case 32: return fft_pass_n<32, R2, R, GI, GO>(N, batch, axis, sign, scale, plan, in, out, st);
    default: return fft_pass_n<0, R2, R, GI, GO>(N, batch, axis, sign, scale, plan, in, out, st);
  }
}

// R2: working type, also the memory type between the passes.
template <typename R2, typename R, typename G>
static edb_status dft3d_t(int N, int batch, const G *in, G *out, int inverse, cudaStream_t st) {
  if (N < 1 || N > FFT_MAXN) return fail(EDB_EINVAL, "dft3d: N out of range [1,64]");
  const int sign = inverse ? +1 : -1;
  const FftPlan plan = fft_plan(N);
  const R one = (R)1;
  const R scale = inverse ? (R)(1. / ((double)N * N * N)) : one;
  R2 *mid = reinterpret_cast<R2 *>(out);
  EDB_TRY((fft_pass<R2, R, G, R2>(N, batch, 2, sign, one, plan, in, mid, st)));
  EDB_TRY((fft_pass<R2, R, R2, R2>(N, batch, 1, sign, one, plan, mid, mid, st)));
  return fft_pass<R2, R, R2, G>(N, batch, 0, sign, scale, plan, mid, out, st);
}

edb_status launch_dft3d(int N, int batch, const void *d_in, void *d_out, void *d_tmp, int inverse,
                        int fp32, cudaStream_t st) {
  (void)d_tmp;
  if (fp32 == EDB_DFT_DOUBLE_FLOAT)
    return dft3d_t<dfc, double, double2>(N, batch, (const double2 *)d_in, (double2 *)d_out,
                                         inverse, st);
  if (fp32)
    return dft3d_t<float2, float, float2>(N, batch, (const float2 *)d_in, (float2 *)d_out,
                                          inverse, st);
  return dft3d_t<double2, double, double2>(N, batch, (const double2 *)d_in, (double2 *)d_out,
                                           inverse, st);
}

}  // namespace edb
