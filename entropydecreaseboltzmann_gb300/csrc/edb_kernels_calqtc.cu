// Batched FP32 collision sum on the tensor cores (ALIASED mode), for the sizes
// that tc_takes() names.
//
// Work: Q^s_K = sum over visited L of B[L][K] f^s_L f^s_(K-L) for S solves
// sharing the pair table B (see genB32_tc_kernel).  Every product has a weight
// of its own, so the sum itself is no GEMM; but the products are: the outer
// product of a set of f_L with a line of f_M is a rank-1 (complex) matrix, and
// the tensor cores form it at a small part of their rate while the FP32 pipe
// is left with one packed FMA per complex product (weight times product, added)
// in place of three.
//
// Products at FP32 accuracy: each FP32 value is cut into three bf16 parts,
// x = h + m + l exactly (8 significand bits each, by truncation), and one
// tcgen05.mma of K = 16 sums the eight part products h h, h m, h l, m h, m m,
// m l, l h, l m of re re and the eight of -im im (of re im and im re for the
// imaginary part).  Only l l, below 2^-32 of the product, is left out.  Error
// against 64 bits, relative to the largest value: 37 solves of N = 21 7.9e-7
// (calq32_kernel 8.5e-7).
//
// A CTA owns one output plane k1 of SG solves.  Step = (l1 plane, m2 line,
// block v of CL consecutive l3).  The 128 tensor-memory lanes are (k2, c): lane
// k2 CL + c holds l2 = k2 - m2 and l3 = v CL + c, the columns j hold
// m3 = j - v CL, all mod N, so every lane keeps the same outputs
// (k2, k3 = c + j) through the whole sum and its weighted products add up in
// registers.  One tile = one solve's 128 x NC products of a step.
//
// Warps: 0-7 compute (warpgroup h takes solves h, h + 2): read a tile from tensor
// memory, one packed FMA per product with the step's weights, which they load
// once for their solves.  8-11 write the A operand (the parts of f_L, one row
// per lane) to tensor memory: from shared memory an MMA of so few columns would
// be bound by reading A (40 clocks against 16).  12 issues the MMAs.  13 streams
// the weights (one bulk copy per step).  14-15 write the B operand (the parts of
// a line of f_M, repeated so that the rotation by v CL is only an offset) and
// stage the next f_L plane.  Every hand-over is an mbarrier and every wait is
// bounded.
//
// Summation: plain FP32 over 5 N / 2 terms in a lane, then over the CL lanes of
// an output; the result joins a compensated (hi, lo) sum.  No term takes part in
// as many plain additions as in calq32_kernel (4 N), and the error against 64
// bits is below that kernel's at every size.  Relative L2, that kernel -> this
// one (with 4 N terms in a lane): white noise, N = 13 1.63e-7 -> 1.54e-7 (1.83e-7),
// 17 1.87e-7 -> 1.64e-7 (1.94e-7), 31 2.46e-7 -> 1.91e-7 (2.35e-7); BKW with a bump,
// N = 13 5.9e-7 -> 5.1e-7 (6.6e-7), 21 8.5e-7 -> 7.0e-7 (8.3e-7).  The shorter sums
// cost 1.5 to 6% (4096 of N = 13 9.20 -> 9.54 ms, 37 of N = 21 770 -> 806 us).
//
// What bounds it: the hand-overs between the roles and the A rows beside the
// FMAs (a tile of N = 21 takes about 256 clocks an SM, its FMAs 60; an SM with work
// issues in 56% of its cycles, FMA pipe 17%, tensor pipe 12%).  Measured, ms, calq32_kernel's
// plain-load path -> here: 37 solves of N = 21 2.80 -> 0.81, 256 of N = 31 126 -> 34,
// 16 of N = 17 0.82 -> 0.16.
//
// Range: a solve with an infinity or a NaN is NaN throughout, as in calq32_kernel;
// products that overflow before they are weighted see tc_direct.
#include <algorithm>

#include "edb_df.cuh"
#include "edb_internal.cuh"

namespace edb {
namespace {

typedef unsigned long long u64;
constexpr int TC_THREADS = 512;
constexpr int TC_HDR = 1024;
constexpr int MAX_STG = 8;

__device__ __forceinline__ uint32_t s_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// One arrival from the lanes with `on`, by predication: a divergent branch
// around it costs a converged warp about 70 clocks.
__device__ __forceinline__ void mbar_arrive(uint32_t bar, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n"
      " @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}\n" ::"r"(bar),
      "r"((int)on)
      : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase with this parity for at most lim nanoseconds.  When it
// runs out lim becomes 0, and later waits of the thread return after one poll:
// no role leaves its loop early, so nothing ever waits for a role that left.
// `ready`: the outcome of an earlier mbar_try, issued ahead so that its
// latency passes under other work.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, u64 &lim,
                                          bool ready = false) {
  asm volatile(
      "{\n .reg .pred P;\n .reg .u64 t0, t1;\n"
      " setp.ne.b32 P, %3, 0;\n"
      " @P bra DONE_%=;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      " @P bra DONE_%=;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      " @P bra DONE_%=;\n"
      " mov.u64 t0, %%globaltimer;\n"
      "POLL_%=:\n"
      " mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      " @P bra DONE_%=;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      " @P bra DONE_%=;\n"
      " mov.u64 t1, %%globaltimer;\n"
      " sub.u64 t1, t1, t0;\n"
      " setp.lt.u64 P, t1, %0;\n"
      " @P bra POLL_%=;\n"
      " mov.u64 %0, 0;\n"
      "DONE_%=:\n}\n"
      : "+l"(lim)
      : "r"(bar), "r"(parity), "r"((int)ready)
      : "memory");
}
// The same for a role with slack: it sleeps between polls and leaves the issue
// slots and the shared-memory pipe to the others.
__device__ __forceinline__ void mbar_doze(uint32_t bar, uint32_t parity, u64 &lim, uint32_t ns) {
  asm volatile(
      "{\n .reg .pred P;\n .reg .u64 t0, t1;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      " @P bra DONE_%=;\n"
      " mov.u64 t0, %%globaltimer;\n"
      "POLL_%=:\n"
      " nanosleep.u32 %3;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      " @P bra DONE_%=;\n"
      " mov.u64 t1, %%globaltimer;\n"
      " sub.u64 t1, t1, t0;\n"
      " setp.lt.u64 P, t1, %0;\n"
      " @P bra POLL_%=;\n"
      " mov.u64 %0, 0;\n"
      "DONE_%=:\n}\n"
      : "+l"(lim)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
}
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity, u64 lim) {
  mbar_wait(bar, parity, lim);
  return lim != 0;
}

// One bulk copy to shared memory and the bytes its barrier waits for.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint32_t bar, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " @p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %2;\n"
      " @p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
      "[%3];\n}\n" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "r"((int)on)
      : "memory");
}

// ---- tensor memory
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar, bool on) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n"
      " @p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
          bar),
      "r"((int)on)
      : "memory");
}
// D = A B^T, A (128 x 16 bf16) in tensor memory, B (n x 16) in shared memory.
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, u64 bdesc, uint32_t idesc, bool on) {
  asm volatile(
      "{\n .reg .pred p, z;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 z, 0, 0;\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, z;\n}\n" ::"r"(d),
      "r"(a), "l"(bdesc), "r"(idesc), "r"((int)on)
      : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t a, const uint32_t (&w)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::
                   "r"(a),
               "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]),
               "r"(w[7])
               : "memory");
}
// Consecutive columns of this lane, asynchronously: the outputs are the registers
// that the load itself writes, and nothing reads them before tc_wait_ld.
__device__ __forceinline__ void tc_ld8(uint32_t a, uint32_t *x) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]),
        "=r"(x[7])
      : "r"(a));
}
__device__ __forceinline__ void tc_ld16(uint32_t a, uint32_t *x) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]),
        "=r"(x[7]), "=r"(x[8]), "=r"(x[9]), "=r"(x[10]), "=r"(x[11]), "=r"(x[12]), "=r"(x[13]),
        "=r"(x[14]), "=r"(x[15])
      : "r"(a));
}
template <int CH>
__device__ __forceinline__ void tc_ld(uint32_t a, uint32_t *x) {
  tc_ld16(a, x);
  if constexpr (CH == 24) tc_ld8(a + 16, x + 16);
  if constexpr (CH == 32) tc_ld16(a + 16, x + 16);
}
// Completes this thread's loads; the registers pass through so that no use of
// them (packing them into pairs among those) is scheduled before it.
template <int CH>
__device__ __forceinline__ void tc_wait_ld(uint32_t (&x)[CH]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < CH; ++j) asm volatile("" : "+r"(x[j]));
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}\n"
               : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ float2 lds_f2(uint32_t ad, bool on) {  // zero where off
  float2 v;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n"
      " @p ld.shared.v2.f32 {%0, %1}, [%2];\n}\n"
      : "=&f"(v.x), "=&f"(v.y)
      : "r"(ad), "r"((int)on));
  return v;
}
__device__ __forceinline__ void sts_u4(uint32_t ad, uint4 w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ad), "r"(w.x), "r"(w.y), "r"(w.z),
               "r"(w.w)
               : "memory");
}
// (hi, lo) += x, without error in hi + lo but for the rounding of lo.
__device__ __forceinline__ void two_sum(float &hi, float &lo, float x) {
  const float s = hi + x, bb = s - hi;
  lo += (hi - (s - bb)) + (x - bb);
  hi = s;
}
__device__ __forceinline__ float2 upk(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ u64 pk(uint32_t a, uint32_t b) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void fma2(u64 &acc, u64 a, u64 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
// x = h + m + l, each part with at most 8 significand bits, in the upper
// halves of the words (bf16 by truncation).
struct Parts {
  uint32_t h, m, l;
};
__device__ __forceinline__ Parts cut(float x) {
  Parts p;
  p.h = __float_as_uint(x) & 0xffff0000u;
  const float r = x - __uint_as_float(p.h);
  p.m = __float_as_uint(r) & 0xffff0000u;
  p.l = __float_as_uint(r - __uint_as_float(p.m));
  return p;
}
// bf16 pair (first in the lower half) from two upper halves.
__device__ __forceinline__ uint32_t pair(uint32_t a, uint32_t b) {
  return __byte_perm(a, b, 0x7632);
}
// K slots of the A operand (h h h m m m l l) and the B operand (h m l h m l h m).
__device__ __forceinline__ void a_words(float x, uint32_t *w) {
  const Parts p = cut(x);
  w[0] = pair(p.h, p.h);
  w[1] = pair(p.h, p.m);
  w[2] = pair(p.m, p.m);
  w[3] = pair(p.l, p.l);
}
__device__ __forceinline__ uint4 b_words(float x) {
  const Parts p = cut(x);
  const uint32_t hm = pair(p.h, p.m);
  return make_uint4(hm, pair(p.l, p.h), pair(p.m, p.l), hm);
}

}  // namespace

// Geometry of a size: CL l3 values per step, V steps per line, NC columns.
TcGeom tc_geom(int N) {
  TcGeom g;
  const int cmax = std::min(N, 128 / N);
  g.V = (N + cmax - 1) / cmax;
  g.CL = (N + g.V - 1) / g.V;
  g.NC = N <= 16 ? 16 : N <= 24 ? 24 : 32;
  // 8-byte words per staged plane row: CL mod 16, so that the lanes' reads
  // (runs of CL at this pitch) fall on consecutive banks
  g.pitch = g.CL;
  while (g.pitch < N) g.pitch += 16;
  return g;
}

struct TcArgs {
  int N, S, CL, V, pitch, C, NST, FL;  // FL: steps per fold
  int N4;                              // weight columns stored
  int first, end;                      // this launch's solves
  const float *B32;
  const float2 *fin;
  float2 *Q;
  float4 *partial;
  unsigned long long wait_ns;
  int *status;  // set to 1 when a bounded wait ran out
};

template <int NC, int SG>
struct TcCfg {
  static constexpr int NCM = NC <= 16 ? 16 : 32;  // MMA columns (a multiple of 16)
  // tensor-memory columns of a tile: the real columns, then the imaginary ones
  // (the spare MMA columns of the real part are written first, then replaced)
  static constexpr int DC = NC + NCM;
  static constexpr int TP = NC == 16 ? SG : 2;    // tiles per hand-over
  static constexpr int UC = TP * DC;
  static constexpr int AB = 4;                    // A operand buffers (steps)
  static constexpr int AC = AB * SG * 8;
  static constexpr int NU0 = (512 - AC) / UC;
  static constexpr int NU = NU0 > 6 ? 6 : NU0;    // tile units
  static constexpr int CH = NC == 32 ? 16 : NC == 24 ? 24 : 32;  // columns per read of a tile
  // registers of a compute and of a service thread (2 RC + 2 RS = 4 x 128); at 192
  // the largest form spills 76 bytes, at 200 the others' service threads do
  static constexpr int RC = NC == 32 && SG == 4 ? 200 : 192, RS = 256 - RC;
  static constexpr int NPB = NC == 32 ? 1 : 2;    // staged f_L planes
  static constexpr int SB = 128 * NC * 4;         // bytes of a ring stage
  static constexpr int PITCH = NC + 1;            // floats per lane of the fold's staging
  static_assert(NU >= 2, "tensor memory");
  static constexpr int oplen(int N) { return N - 1 + NCM; }  // rows of an operand array
  static constexpr size_t sums(int N) { return (size_t)SG * N * N * 16; }
  static constexpr size_t stage() { return 2u * 128 * PITCH * 4; }
};

// One output (k1, k2, k3) over the planes [P0, P0 + np) of f (one solve), term by
// term with the weight first, in calq32_kernel's form.  Products are formed
// before they are weighted, and one that leaves FP32's range makes its output
// infinite or no number; where the inputs are finite it is summed again here,
// since its weighted terms may be in range (37 of N = 21: 0.81 ms, 2.4 with one such
// solve, 8.9 with all of them; a solve with a NaN costs nothing).
static __device__ float4 tc_direct(const TcArgs &a, const float2 *f, int k1, int k2, int k3, int P0,
                                   int np) {
  const int N = a.N, NN = N * N, plo = k1 / 2;
  float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int p = P0; p < P0 + np; ++p) {
    const int l1 = p <= plo ? p : k1 + 1 + (p - plo - 1), m1 = k1 < l1 ? k1 - l1 + N : k1 - l1;
    for (int m2 = 0; m2 < N; ++m2) {
      const int l2 = k2 < m2 ? k2 - m2 + N : k2 - m2;
      const float2 *fl = f + l1 * NN + l2 * N, *fm = f + m1 * NN + m2 * N;
      const float *line = a.B32 + ((long long)(k1 * c32_maxlist(N) + p) * N + m2) * a.V * a.N4 * 128;
      float ax = 0.f, ay = 0.f, bx = 0.f, by = 0.f;  // sums of f_l.re and of f_l.im
      for (int l3 = 0; l3 < N; ++l3) {
        const int v = l3 / a.CL, c = l3 - v * a.CL, j = k3 < c ? k3 - c + N : k3 - c;
        const float w = line[((long long)(v * (a.N4 / 4) + j / 4) * 128 + k2 * a.CL + c) * 4 + j % 4];
        const float2 x = fl[l3], y = fm[k3 < l3 ? k3 - l3 + N : k3 - l3];
        const float qx = w * y.x, qy = w * y.y;
        ax = __fmaf_rn(x.x, qx, ax);
        ay = __fmaf_rn(x.x, qy, ay);
        bx = __fmaf_rn(x.y, qx, bx);
        by = __fmaf_rn(x.y, qy, by);
      }
      two_sum(h.x, h.y, ax - by);
      two_sum(h.z, h.w, ay + bx);
    }
  }
  return h;
}
static __device__ __forceinline__ bool tc_finite(float4 h) {
  return isfinite(h.x + h.y) && isfinite(h.z + h.w);
}
// The CTA's sums that are not finite though their solve's inputs are, again.
// Everything is derived from the block's index anew, so that nothing is kept in
// registers for this through the roles' loops.
template <int SG>
static __device__ __forceinline__ void tc_again(const TcArgs &a, float4 *sums) {
  int block, tid;
  asm volatile("mov.u32 %0, %%ctaid.x;\n mov.u32 %1, %%tid.x;" : "=r"(block), "=r"(tid));
  const int N = a.N, NN = N * N, groups = (a.end - a.first + SG - 1) / SG, grp = block % groups;
  const int chunk = block / groups % a.C, k1 = block / groups / a.C;
  const int s0 = a.first + grp * SG, ns = min(SG, a.end - s0);
  const int nlist = c32_nlist(N, k1), ppc = (nlist + a.C - 1) / a.C;
  const int P0 = min(nlist, chunk * ppc), np = min(nlist, P0 + ppc) - P0;
  for (int s = 0; s < ns; ++s) {
    const float2 *f = a.fin + (long long)(s0 + s) * NN * N;
    bool in = true;
    for (int e = tid; e < NN * N; e += TC_THREADS) in &= isfinite(f[e].x) && isfinite(f[e].y);
    if (__syncthreads_or(!in)) continue;
    for (int e = tid; e < NN; e += TC_THREADS)
      if (!tc_finite(sums[s * NN + e]))
        sums[s * NN + e] = tc_direct(a, f, k1, e / N, e % N, P0, np);
  }
  __syncthreads();
}

// Barriers in the header (8 bytes each)
enum {
  BF = 0,             // weights landed [MAX_STG]
  BE = BF + MAX_STG,  // weights read [MAX_STG]
  AF = BE + MAX_STG,  // A operand written [4]
  AE = AF + 4,        // A operand read [4]
  OF = AE + 4,        // B operand written [2]
  OE = OF + 2,        // B operand read [2]
  DF = OE + 2,        // tile unit ready [6]
  DE = DF + 6,        // tile unit read [6]
  PF = DE + 6,        // f_L plane staged [2]
  PE = PF + 2,        // f_L plane read [2]
  XD = PE + 2,        // all MMAs done
  NBAR = XD + 1
};

template <int NC, int SG>
__global__ void __launch_bounds__(TC_THREADS, 1) calqtc_kernel(const TcArgs a) {
  using Cfg = TcCfg<NC, SG>;
  constexpr int NU = Cfg::NU, NCM = Cfg::NCM, TP = Cfg::TP, AB = Cfg::AB;
  constexpr int NPB = Cfg::NPB;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sb = s_addr(smem);
  auto bar = [&](int i) { return sb + 8u * i; };
  int *tm_slot = reinterpret_cast<int *>(smem + 8 * NBAR);
  int *issued = tm_slot + 1;  // weight copies issued
  const int N = a.N, CL = a.CL, V = a.V, C = a.C;
  const int NN = N * N;
  const long long NQ = (long long)NN * N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // shared memory: header, weight ring, compensated sums, fold staging, f_L
  // planes, B operands
  const uint32_t o_sum = TC_HDR + (uint32_t)a.NST * Cfg::SB;
  const uint32_t o_stage = o_sum + (uint32_t)Cfg::sums(N);
  const uint32_t ring = sb + TC_HDR;
  const uint32_t planes = sb + o_stage + (uint32_t)Cfg::stage();
  const uint32_t PSZ = (uint32_t)N * a.pitch * 8u;  // a staged plane of one solve
  const uint32_t OLEN = (uint32_t)Cfg::oplen(N) * 16u;  // an operand array
  const uint32_t OPS = 3u * OLEN;                       // im, re, -im arrays of one solve
  const uint32_t ops = (planes + (uint32_t)(NPB * SG) * PSZ + 127u) & ~127u;
  u64 lim = a.wait_ns;

  // CTA -> (solve group, k1, chunk): groups fastest, so that the CTAs in
  // flight read the same weights at about the same time
  const int groups = (a.end - a.first + SG - 1) / SG;
  const int grp = blockIdx.x % groups;
  const int rest = blockIdx.x / groups;
  const int chunk = rest % C, k1 = rest / C;
  const int s0 = a.first + grp * SG;
  const int ns = min(SG, a.end - s0);
  const int nlist = c32_nlist(N, k1), plo = k1 / 2;
  const int ppc = (nlist + C - 1) / C;
  const int P0 = min(nlist, chunk * ppc), np = min(nlist, P0 + ppc) - P0;
  auto plane_l1 = [&](int p) { return p <= plo ? p : k1 + 1 + (p - plo - 1); };
  const int lines = np * N, total = lines * V;  // m2 lines and steps

  if (tid == 0) {
    for (int i = 0; i < MAX_STG; ++i) {
      mbar_init(bar(BF + i), 1);
      mbar_init(bar(BE + i), 8);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(bar(AF + i), 4);
      mbar_init(bar(AE + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(OF + i), 2);
      mbar_init(bar(OE + i), 1);
      mbar_init(bar(PF + i), 2);
      mbar_init(bar(PE + i), 4);
    }
    for (int i = 0; i < 6; ++i) {
      mbar_init(bar(DF + i), 1);
      mbar_init(bar(DE + i), 8);
    }
    mbar_init(bar(XD), 1);
    *issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     s_addr(tm_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = (uint32_t)*tm_slot;
  const uint32_t tmA = tm + NU * Cfg::UC;

  if (warp < 8) {
    // ------------------------------------------------------------ compute
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::RC));
    // warpgroup h takes solves h, h + 2, ..., all columns
    const int h = warp >> 2, q = warp & 3;
    constexpr int SW = SG / 2, TW = TP / 2;  // tiles of a step, of a unit
    constexpr int CH = Cfg::CH, K = 2 * NC / CH;  // a tile comes in K reads
    constexpr int P1 = Cfg::PITCH;
    const uint32_t myB = ring + (uint32_t)(q * 32 + lane) * 16u;
    const uint32_t lastB = (uint32_t)(a.N4 / 4 - 1) * 2048u;  // group NC / 4 - 1, or one less
    const uint32_t d0 = tm + ((uint32_t)(q * 32) << 16) + h * Cfg::DC;
    float *stage = reinterpret_cast<float *>(smem + o_stage) + h * 128 * P1;
    float4 *sums = reinterpret_cast<float4 *>(smem + o_sum);  // (hi, lo) of re and im
    for (int e = tid; e < SG * NN; e += 256) sums[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    u64 acc[SW][NC], b[NC / 2];  // re then im pairs; weights
    uint32_t x[2][CH];
#pragma unroll
    for (int s = 0; s < SW; ++s)
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[s][j] = 0ull;
    auto load_b = [&](int stg) {
#pragma unroll
      for (int j = 0; j < NC / 4; ++j)
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];"
                     : "=l"(b[2 * j]), "=l"(b[2 * j + 1])
                     : "r"(myB + (uint32_t)(stg * Cfg::SB) + (j == NC / 4 - 1 ? lastB : j * 2048u)));
    };
    // read k of this warpgroup's tile i of unit u
    auto read = [&](int u, int i, int k, uint32_t (&d)[CH]) {
      tc_ld<CH>(d0 + (uint32_t)(u * Cfg::UC + 2 * i * Cfg::DC + k * CH), d);
    };
    constexpr bool even = (SW * K) % 2 == 0;
    int st = 0, sp = 0, du = 0, dp = 0, fc = a.FL;
    bool rd = false, rb = false;  // outcomes of the polls ahead
    // first read of the next unit (after the last step: of a unit that does not
    // come, without waiting; every read and load is unconditional so that no
    // register is kept for the path without it)
    auto first = [&](uint32_t (&d)[CH], bool last) {
      mbar_wait(bar(DF + du), dp, lim, rd | last);
      tc_fence_after();
      read(du, 0, 0, d);
    };
    auto poll_unit = [&] {  // the unit after du
      const int un = du + 1 == NU ? 0 : du + 1;
      rd = mbar_try(bar(DF + un), un == 0 ? dp ^ 1 : dp);
    };
    if (total > 0) {
      mbar_wait(bar(BF), 0, lim);
      load_b(0);
      first(x[0], false);
      poll_unit();
    }
    for (int i = 0; i < total; ++i) {
      const bool last = i + 1 == total;
      const int stc = st;  // this step's stage
      if (++st == a.NST) {
        st = 0;
        sp ^= 1;
      }
#pragma unroll
      for (int s = 0; s < SW; ++s) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          uint32_t (&cur)[CH] = x[(s * K + k) & 1], (&nxt)[CH] = x[(s * K + k + 1) & 1];
          // the next read is on its way while this one is used
          tc_wait_ld(cur);
          if (k + 1 < K) {
            read(du, s % TW, k + 1, nxt);
          } else if (s % TW + 1 < TW) {
            read(du, s % TW + 1, 0, nxt);
          } else {
            tc_fence_before();
            mbar_arrive(bar(DE + du), lane == 0);
            if (++du == NU) {
              du = 0;
              dp ^= 1;
            }
            if (even || s + 1 < SW) {
              first(nxt, s + 1 == SW && last);
              poll_unit();
            }
          }
          if (k == K - 1 && s == SW - 1) rb = mbar_try(bar(BF + st), sp);
#pragma unroll
          for (int j = 0; j < CH / 2; ++j) {
            const int c = k * (CH / 2) + j;
            fma2(acc[s][c], b[c % (NC / 2)], pk(cur[2 * j], cur[2 * j + 1]));
          }
        }
        // the step's weights are in the registers of every lane, and lane 0 saw
        // them land
        if (s == 0) {
          __syncwarp();
          mbar_arrive(bar(BE + stc), lane == 0 && lim != 0);
        }
      }
      if (!even) {
        first(x[0], last);
        poll_unit();
      }
      mbar_wait(bar(BF + st), sp, lim, rb | last);
      load_b(st);
      if (--fc == 0 || i + 1 == total) {
        // fold: the lanes of an output are added, then joined to its
        // compensated (hi, lo) sum.  The read ahead is completed first: after
        // the last step nothing else does, and its registers are free for the
        // code below.
        fc = a.FL;
        tc_wait_ld(x[0]);
#pragma unroll
        for (int s = 0; s < SW; ++s) {
          float *own = reinterpret_cast<float *>(sums + ((s / TW) * TP + (s % TW) * 2 + h) * NN);
#pragma unroll
          for (int c2 = 0; c2 < 2; ++c2) {
            float *row = stage + (q * 32 + lane) * P1;
#pragma unroll
            for (int j = 0; j < NC / 2; ++j) {
              const float2 y = upk(acc[s][c2 * (NC / 2) + j]);
              row[2 * j] = y.x;
              row[2 * j + 1] = y.y;
              acc[s][c2 * (NC / 2) + j] = 0ull;
            }
            asm volatile("bar.sync %0, 128;" ::"r"(2 + h) : "memory");
            // warp q: outputs k2 = q, q + 4, ..., UR at a time; lane k3
            if (lane < N) {
              constexpr int UR = NC == 24 ? 6 : 4;  // a warp has up to NC / 4 of them
              for (int k0 = q; k0 < N; k0 += 4 * UR) {
                u64 y[UR / 2] = {};  // of two outputs each
                const float *y0[UR];
#pragma unroll
                for (int u = 0; u < UR; ++u) y0[u] = stage + min(k0 + 4 * u, N - 1) * CL * P1;
                int j = lane;
                for (int c = 0; c < CL; ++c) {
#pragma unroll
                  for (int u = 0; u < UR / 2; ++u)
                    y[u] = df::add2(y[u], pk(__float_as_uint(y0[2 * u][c * P1 + j]),
                                             __float_as_uint(y0[2 * u + 1][c * P1 + j])));
                  j = j == 0 ? N - 1 : j - 1;
                }
#pragma unroll
                for (int u = 0; u < UR; ++u) {
                  const int k2 = k0 + 4 * u;
                  if (k2 < N) {
                    float2 *hl = reinterpret_cast<float2 *>(own + 4 * (k2 * N + lane) + 2 * c2);
                    const float2 yy = upk(y[u / 2]);
                    float2 t = *hl;
                    two_sum(t.x, t.y, u & 1 ? yy.y : yy.x);
                    *hl = t;
                  }
                }
              }
            }
            asm volatile("bar.sync %0, 128;" ::"r"(2 + h) : "memory");
          }
        }
      }
    }
  } else if (warp < 12) {
    // ------------------------------------------------------- A operand rows
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::RS));
    const int q = warp - 8;
    const int r = q * 32 + lane;
    const bool row_ok = r < N * CL;
    const int k2 = row_ok ? r / CL : 0, c = row_ok ? r % CL : 0;
    const uint32_t ta = tmA + ((uint32_t)(q * 32) << 16);
    int ab = 0, ap = 1, pb = 0, pp = 0;
    for (int p = 0; p < np; ++p) {
      mbar_wait(bar(PF + pb), pp, lim);
      const uint32_t pl = planes + (uint32_t)(pb * SG) * PSZ;
      int l2 = k2;
      for (int m2 = 0; m2 < N; ++m2) {
        const uint32_t rowa = pl + (uint32_t)(l2 * a.pitch + c) * 8u;
        for (int v = 0; v < V; ++v) {
          const bool ok = row_ok && v * CL + c < N;
          float2 f[SG];
#pragma unroll
          for (int s = 0; s < SG; ++s) {
            f[s] = lds_f2(rowa + (uint32_t)s * PSZ + (uint32_t)(v * CL) * 8u, ok);
          }
          mbar_doze(bar(AE + ab), ap, lim, 100);
          tc_fence_after();
#pragma unroll
          for (int s = 0; s < SG; ++s) {
            uint32_t w[8];
            a_words(f[s].x, w);
            a_words(f[s].y, w + 4);
            tc_st8(ta + (uint32_t)((ab * SG + s) * 8), w);
          }
          tc_wait_st();
          tc_fence_before();
          mbar_arrive(bar(AF + ab), lane == 0);
          if (++ab == AB) {
            ab = 0;
            ap ^= 1;
          }
        }
        l2 = l2 == 0 ? N - 1 : l2 - 1;
      }
      __syncwarp();
      mbar_arrive(bar(PE + pb), lane == 0);
      if (++pb == NPB) {
        pb = 0;
        pp ^= 1;
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::RS));
    if (warp == 12) {
      // ---------------------------------------------------------- MMA issue
      // The whole warp runs the loop and one lane's MMAs are predicated: in a
      // single-lane loop a wait took three times as long and an MMA seven times
      const bool el = elect_one();
      constexpr uint32_t idesc =
          (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NCM >> 3) << 17) | (8u << 24);
      // K-major, no swizzle: rows 16 bytes apart, 8-row groups 128 bytes
      // apart, the two K halves one operand array apart
      const u64 dbase = ((u64)(OLEN >> 4) << 16) | ((u64)(128 >> 4) << 32) | (1ull << 46);
      int ab = 0, ap = 0, ob = 0, op = 0, du = 0, dp = 1;
      bool ra = false, rd = false;
      for (int i = 0; i < lines; ++i) {
        mbar_wait(bar(OF + ob), op, lim);
        for (int v = 0; v < V; ++v) {
          mbar_wait(bar(AF + ab), ap, lim, ra);
          const uint32_t x0 = v == 0 ? 0u : (uint32_t)(N - v * CL) * 16u;
#pragma unroll
          for (int g = 0; g < SG / TP; ++g) {
            mbar_wait(bar(DE + du), dp, lim, rd);
            tc_fence_after();
#pragma unroll
            for (int t = 0; t < TP; ++t) {
              const int s = g * TP + t;
              const uint32_t o = ops + (uint32_t)(ob * SG + s) * OPS + x0;
              const uint32_t d = tm + du * Cfg::UC + t * Cfg::DC;
              const uint32_t ad = tmA + (uint32_t)((ab * SG + s) * 8);
              tc_mma(d, ad, dbase | (u64)(((o + OLEN) >> 4) & 0x3fff), idesc, el);
              tc_mma(d + NC, ad, dbase | (u64)((o >> 4) & 0x3fff), idesc, el);
            }
            tc_commit(bar(DF + du), el);
            if (++du == NU) {
              du = 0;
              dp ^= 1;
            }
            rd = mbar_try(bar(DE + du), dp);
          }
          tc_commit(bar(AE + ab), el);
          if (++ab == AB) {
            ab = 0;
            ap ^= 1;
          }
          ra = mbar_try(bar(AF + ab), ap);
        }
        tc_commit(bar(OE + ob), el);
        ob ^= 1;
        op ^= (ob == 0);
      }
      // every MMA and every commit has landed before the block leaves; one that
      // has not is reported as a wait that ran out
      tc_commit(bar(XD), el);
      if (!mbar_poll(bar(XD), 0, DRAIN_LIMIT_NS)) lim = 0;
    } else if (warp == 13) {
      // ------------------------------------------------------ weight stream
      const char *src = reinterpret_cast<const char *>(a.B32) +
                        (long long)(k1 * c32_maxlist(N) + P0) * N * V * a.N4 * 512;
      const uint32_t bytes = (uint32_t)a.N4 * 512u;  // of a step's weights
      int st = 0, sp = 1, n = 0;
      for (int i = 0; i < total; ++i) {
        mbar_doze(bar(BE + st), sp, lim, 100);
        // nothing more is issued once a wait ran out: the stage's last copy
        // may still be landing
        const bool on = lane == 0 && lim != 0;
        bulk_load(ring + (uint32_t)(st * Cfg::SB), src + (long long)i * bytes, bytes,
                  bar(BF + st), on);
        n += on;
        if (++st == a.NST) {
          st = 0;
          sp ^= 1;
        }
      }
      if (lane == 0) *issued = n;
    } else {
      // ------------------------------------- B operand lines, next f_L plane
      const int w = warp - 14;
      constexpr int SH = (SG + 1) / 2;  // solves of one of the two warps
      const float2 *base = a.fin + (long long)s0 * NQ;
      const int len = Cfg::oplen(N);
      const bool in = lane < N;
      float2 fm[SH], fn[SH];
      auto line = [&](float2 (&f)[SH], int l1, int l2) {
#pragma unroll
        for (int i = 0; i < SH; ++i) {
          const int s = w + 2 * i;
          f[i] = make_float2(0.f, 0.f);
          if (s < ns && in) f[i] = __ldg(base + (long long)s * NQ + (l1 * NN + l2 * N + lane));
        }
      };
      auto put = [&](const float2 (&f)[SH], int buf, int l2) {
#pragma unroll
        for (int i = 0; i < SH; ++i) {
          const int s = w + 2 * i;
          if (s < SG && in)
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(
                             planes + (uint32_t)(buf * SG + s) * PSZ +
                             (uint32_t)(l2 * a.pitch + lane) * 8u),
                         "f"(f[i].x), "f"(f[i].y)
                         : "memory");
        }
      };
      // a whole plane, four rows on their way at a time
      auto whole = [&](int l1, int buf) {
        for (int l2 = 0; l2 < N; l2 += 4) {
          float2 f[4][SH];
#pragma unroll
          for (int i = 0; i < 4; ++i) line(f[i], l1, min(l2 + i, N - 1));
#pragma unroll
          for (int i = 0; i < 4; ++i) put(f[i], buf, min(l2 + i, N - 1));
        }
        __syncwarp();
        mbar_arrive(bar(PF + buf), lane == 0);
      };
      auto m1_of = [&](int p) {
        const int m1 = k1 - plane_l1(P0 + p);
        return m1 < 0 ? m1 + N : m1;
      };
      if (np > 0) {
        whole(plane_l1(P0), 0);
        line(fm, m1_of(0), 0);
      }
      int ob = 0, op = 1;
      for (int p = 0; p < np; ++p) {
        const bool more = p + 1 < np;
        const int l1n = more ? plane_l1(P0 + p + 1) : 0;
        const int m1 = m1_of(p);
        for (int m2 = 0; m2 < N; ++m2) {
          if (NPB == 2 && more) line(fn, l1n, m2);
          mbar_doze(bar(OE + ob), op, lim, 200);
#pragma unroll
          for (int i = 0; i < SH; ++i) {
            const int s = w + 2 * i;
            if (s < SG && in) {
              const uint4 wr = b_words(fm[i].x), wi = b_words(fm[i].y);
              const uint4 wn = make_uint4(wi.x ^ 0x80008000u, wi.y ^ 0x80008000u,
                                          wi.z ^ 0x80008000u, wi.w ^ 0x80008000u);
              const uint32_t o = ops + (uint32_t)(ob * SG + s) * OPS;
              for (int y = lane; y < len; y += N) {
                const uint32_t ad = o + (uint32_t)y * 16u;
                sts_u4(ad, wi);
                sts_u4(ad + OLEN, wr);
                sts_u4(ad + 2 * OLEN, wn);
              }
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          mbar_arrive(bar(OF + ob), lane == 0);
          ob ^= 1;
          op ^= (ob == 0);
          // the next line of f_M, one line ahead
          if (m2 + 1 < N)
            line(fm, m1, m2 + 1);
          else if (more)
            line(fm, m1_of(p + 1), 0);
          if (NPB == 2 && more) {
            if (m2 == 0 && p > 0) mbar_wait(bar(PE + ((p + 1) & 1)), ((p - 1) >> 1) & 1, lim);
            put(fn, (p + 1) & 1, m2);
          }
        }
        if (NPB == 2) {
          __syncwarp();
          mbar_arrive(bar(PF + ((p + 1) & 1)), lane == 0 && more);
        } else if (more) {
          mbar_wait(bar(PE), p & 1, lim);
          whole(l1n, 0);
        }
      }
    }
  }
  __syncwarp();
  // back to the launch's share each: what follows is all warps' code, and at a
  // service thread's share it spills, which costs the loops above 2%
  if (warp < 8)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 128;");
  else
    asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
  const bool aborted = __syncthreads_or(lim == 0) != 0;
  if (aborted) {
    if (tid == 0) {
      atomicExch(a.status, 1);
      // the last copy issued into each stage may still be landing
      const int n = *issued;
      for (int i = max(0, n - a.NST); i < n; ++i)
        mbar_poll(bar(BF + i % a.NST), (uint32_t)((i / a.NST) & 1), DRAIN_LIMIT_NS);
    }
  } else {
    float4 *sums = reinterpret_cast<float4 *>(smem + o_sum);
    bool odd = false;
    for (int e = tid; e < ns * NN; e += TC_THREADS) odd |= !tc_finite(sums[e]);
    if (__syncthreads_or(odd)) tc_again<SG>(a, sums);
    for (int e = tid; e < ns * NN; e += TC_THREADS) {
      const int s = e / NN, k23 = e - s * NN;
      const float4 h = sums[e];
      const long long o = (long long)(s0 + s) * NQ + (long long)k1 * NN + k23;
      if (C == 1)
        a.Q[o] = make_float2(h.x + h.y, h.z + h.w);
      else
        a.partial[(long long)chunk * a.S * NQ + o] = make_float4(h.x, h.z, h.y, h.w);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tm) : "memory");
}

template <int NC, int SG>
static edb_status launch_tc(const TcArgs &args, int first, int end, cudaStream_t st) {
  using Cfg = TcCfg<NC, SG>;
  if (first >= end) return EDB_OK;
  TcArgs a = args;
  a.first = first;
  a.end = end;
  auto kern = calqtc_kernel<NC, SG>;
  static const cudaError_t configured =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (configured != cudaSuccess) return cuda_fail(configured, "cudaFuncSetAttribute(calqtc)");
  const size_t fixed = TC_HDR + Cfg::sums(a.N) + Cfg::stage() +
                       (size_t)Cfg::NPB * SG * a.N * a.pitch * 8 + 256 +
                       2u * SG * 3u * (size_t)Cfg::oplen(a.N) * 16;
  a.NST = (int)std::min<size_t>(MAX_STG, (227 * 1024 - fixed) / Cfg::SB);
  // at least half of an SM's shared memory: one CTA per SM holds all of its
  // tensor memory
  const size_t bytes = std::max<size_t>(fixed + (size_t)a.NST * Cfg::SB, 120 * 1024);
  const long long blocks = (long long)((end - first + SG - 1) / SG) * a.N * a.C;
  kern<<<(unsigned)blocks, TC_THREADS, bytes, st>>>(a);
  EDB_LAUNCHED();
  return EDB_OK;
}

// Solves per CTA: 4 for the first tc_fours() solves and 2 for the others, in a
// launch of their own, by the number of CTA waves.  A wave of CTAs of 2 takes
// 0.67 of one of 4 at 16 weight columns and 0.63 above (N = 13 74 | 109 us, 21
// 311 | 492, 31 1476 | 2285): 37 x N = 21 944 us in CTAs of 4 (210 of them on 152
// SMs), 887 in CTAs of 2, 795 as 28 + 9; 17 x N = 31 4.44 -> 2.86 ms, 30 x N = 25
// 1.90 -> 1.59 ms.  A second launch has to gain 3% and its start: over many waves
// the CTAs drift apart, and a last one that is part full costs less (500 x N = 21
// 8.45 ms, 8.55 as 492 + 8).
// Each wave of fours given up costs at least 0.26 of a wave and all of them
// together gain less than the last part-full one, so only the last few waves'
// groups are tried: 4096 x N = 13 11.5 -> 8 us of host time a call, 40,000 58 -> 9.
int tc_fours(int S, int N, int C, int sms) {
  const double two = tc_geom(N).NC == 16 ? 0.67 : 0.63;
  const long long per = (long long)N * C;
  auto waves = [&](long long groups) { return (double)((groups * per + sms - 1) / sms); };
  const int all = (S + 3) / 4, wave = (int)(sms / per) + 1;  // groups, at least a wave's
  int four = S;
  double best = 1e30;
  for (int g4 = all; g4 >= std::max(0, all - 8 * wave); --g4) {
    const int n4 = std::min(S, 4 * g4), n2 = S - n4;
    double t = waves(g4) + two * waves((n2 + 1) / 2);
    if (n2 > 0 && n4 > 0) t = 1.03 * t + 0.02;
    if (t < best - 1e-9) {
      best = t;
      four = n4;
    }
  }
  return four;
}

edb_status launch_calqtc(int N, int S, const float *d_B32, const float2 *d_fin, float2 *d_Q, int C,
                         float4 *d_partial, cudaStream_t st) {
  const TcGeom g = tc_geom(N);
  TcArgs a;
  a.N = N;
  a.S = S;
  a.CL = g.CL;
  a.V = g.V;
  a.pitch = g.pitch;
  a.C = C;
  a.FL = 5 * N / 2;
  a.B32 = d_B32;
  a.fin = d_fin;
  a.Q = d_Q;
  a.partial = d_partial;
  a.wait_ns = wait_limit_ns();
  EDB_TRY(calq32_status_ptr(&a.status));
  a.NST = 0;
  a.N4 = (N + 3) / 4 * 4;
  const int four = tc_fours(S, N, C, device_sm_count());
#define EDB_TC(NC)                                \
  EDB_TRY((launch_tc<NC, 4>(a, 0, four, st)));    \
  return launch_tc<NC, 2>(a, four, S, st)
  switch (g.NC) {
    case 16: EDB_TC(16);
    case 24: EDB_TC(24);
    default: EDB_TC(32);
  }
#undef EDB_TC
}

}  // namespace edb
