// Free streaming in x for spatially inhomogeneous use of the collision step.
//
// The reference solves the space-homogeneous equation only (BKW.h integrates
// df/dt = Q(f) for one velocity distribution).  The inhomogeneous equation
//   df/dt + v1 df/dx = Q(f)
// on a periodic 1-D x grid of C cells splits into a transport step (this
// kernel) and one homogeneous collision step per cell (the batched solver,
// one solve per cell), e.g. Strang: transport dt/2, collide dt, transport dt/2.
//
// Layout: cells-major, f[c][v] with v the N^3 velocity grid points
// v_d = -R + i_d h, h = 2R/N (row-major [i1][i2][i3], as BKW.h:124-133), so
// one cell's distribution is the contiguous N^3 block a batched solve reads.
//
// Scheme: semi-Lagrangian with linear interpolation.  The foot of the
// characteristic through x_c is x_c - v1 dt, s = v1 dt / dx cells upstream,
// s = n + theta with n = floor(s):
//   f_out[c][v] = (1 - theta) f[(c - n) mod C][v] + theta f[(c - n - 1) mod C][v].
// For each velocity the weights sum to one over the periodic grid, so the
// total of every velocity slice (and with it mass, momentum and energy) is
// kept exactly up to rounding; the weights are non-negative, so f >= 0 is
// kept; theta = 0 (an integer shift) is exact.  One read of two neighbours and
// one write per entry, coalesced along v.
#include <math.h>

#include <algorithm>
#include <cmath>

#include "edb_internal.cuh"

namespace edb {

// A block owns one velocity index i1 and every G-th cell.  The shift and weights
// depend on i1 only, and their FP64 division and floor cost more than an entry's
// own arithmetic (FP64 is what bounds this kernel, not its bytes), so thread 0
// evaluates them once a block.  Evaluated per entry, 256
// cells x N = 16 took 59.6 us (now 12.0), 512 x N = 32 612 us (85).
__global__ void transport_x_kernel(int C, int N, int G, double R, double dx, double dt,
                                   const double *__restrict__ f, double *__restrict__ out) {
  const int NN = N * N;
  const long long NQ = (long long)NN * N;
  const int i1 = (int)(blockIdx.x % N);
  __shared__ double sh_theta;
  __shared__ int sh_n;
  if (threadIdx.x == 0) {
    const double h = 2.0 * R / N;
    const double v1 = -R + i1 * h;
    const double s = v1 * dt / dx;
    const double fl = floor(s);
    sh_theta = s - fl;
    // n mod C as a non-negative shift (|n| may exceed C for large dt)
    long long n = (long long)fl % C;
    sh_n = (int)(n < 0 ? n + C : n);
  }
  __syncthreads();
  const double theta = sh_theta, keep = 1.0 - theta;
  const int n = sh_n;
  for (int c = (int)(blockIdx.x / N); c < C; c += G) {
    const int c0 = c >= n ? c - n : c - n + C;
    const int c1 = c0 == 0 ? C - 1 : c0 - 1;
    const double *fa = f + c0 * NQ + (long long)i1 * NN, *fb = f + c1 * NQ + (long long)i1 * NN;
    double *o = out + c * NQ + (long long)i1 * NN;
    for (int e = threadIdx.x; e < NN; e += blockDim.x)
      o[e] = keep * __ldg(fa + e) + theta * __ldg(fb + e);
  }
}

edb_status launch_transport_x(int C, int N, double R, double Lx, double dt, const double *d_f,
                              double *d_out, cudaStream_t st) {
  // about eight blocks an SM
  const int G = std::max(1, std::min(C, 8 * device_sm_count() / N));
  const int threads = std::min(256, (N * N + 31) / 32 * 32);
  transport_x_kernel<<<(unsigned)(N * G), threads, 0, st>>>(C, N, G, R, Lx / C, dt, d_f, d_out);
  EDB_LAUNCHED();
  return EDB_OK;
}

}  // namespace edb

using namespace edb;

extern "C" edb_status edb_cells_transport_x_device(int C, int N, double R, double Lx, double dt,
                                                   const double *d_f, double *d_out,
                                                   void *stream) {
  if (C < 1 || N < 3 || N > 64 || !(R > 0) || !(Lx > 0) || !std::isfinite(dt))
    return fail(EDB_EINVAL, "transport: bad argument");
  if (!d_f || !d_out) return fail(EDB_EINVAL, "transport: null device pointer");
  if (d_f == d_out) return fail(EDB_EINVAL, "transport: input and output must differ");
  EDB_TRY(ensure_device());
  return launch_transport_x(C, N, R, Lx, dt, d_f, d_out, (cudaStream_t)stream);
}
