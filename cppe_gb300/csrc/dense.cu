// Small direct-summation systems in FP64: the operator as a dense matrix, and
// the whole PCG of the smallest ones in one thread block.
//
// A pair of the direct sum takes 30 to 60 FP64 instructions, an entry of the
// matrix one: 999 sites take 24 us an apply (15 us of multiply-adds at 1.96 FP64
// lane-operations per clock and SM) against 88 us of k_p2p64 and k_finish; 60
// sites 6 us against 51.  The matrix is built once per system, each pair once
// (66 us at 999 sites).  DENSE_MAX: up to there build and apply together cost
// what one pair-kernel apply does, so that a first call of one apply is no slower,
// the matrix (75 MB) stays in L2 and one cluster takes the iteration's vector part;
// at 1,998 sites they take 243 + 80 us against 144 (a solve of 14 applies would still
// gain), at 2,997 536 + 162 us against 206.  The matrices of all systems share
// DENSE_POOL bytes.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "system.h"

namespace cg {

namespace coop = cooperative_groups;

constexpr int DENSE_BLOCK   = 128;  // threads per site (three rows) of the product
constexpr int STEP_BLOCK    = 128;  // sites per block of the iteration's vector part,
constexpr int STEP_CLUSTER  = 8;    // which is one cluster
static_assert(STEP_BLOCK * STEP_CLUSTER >= DENSE_MAX, "one cluster per system");
static_assert(STEP_BLOCK == 128 && STEP_CLUSTER == 8, "one warp's value per lane");
constexpr int SMALL_THREADS = (3 * SMALL_MAX + 31) / 32 * 32;

// -T (row-major, 3n x 3n; T is symmetric, its diagonal blocks zero), zero where the
// row's site excludes the column's: B of BMatrix (src/core/bmatrix.cc:9-40) without
// alpha^-1, which the product adds last (a sum that starts from the large diagonal
// term rounds every further term to it).  Thread per unordered pair.
__global__ void k_dense_build(int n, const double4_32a* __restrict__ pos,
                              const int* __restrict__ eptr, const int* __restrict__ eidx, int damp,
                              double damping, double* __restrict__ B) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)n * (n + 1) / 2) return;
  // t = i (i + 1) / 2 + j, j <= i
  int i = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((long)i * (i + 1) / 2 > t) --i;
  while ((long)(i + 1) * (i + 2) / 2 <= t) ++i;
  const int j     = (int)(t - (long)i * (i + 1) / 2);
  const size_t N3 = 3 * (size_t)n;
  double b[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  bool zij = false, zji = false;
  if (i != j) {
    for (int e = eptr[i]; e < eptr[i + 1]; ++e) zij |= eidx[e] == j;
    for (int e = eptr[j]; e < eptr[j + 1]; ++e) zji |= eidx[e] == i;
    const double4_32a pi = pos[i], pj = pos[j];
    const double r[3] = {pi.x - pj.x, pi.y - pj.y, pi.z - pj.z};
    const double r2   = fma(r[0], r[0], fma(r[1], r[1], r[2] * r[2]));
    double G[2];
    radial<double, 2>(r2, damp ? damping * pi.w * pj.w : 0.0, G);
    const double g[3] = {r[0] * G[1], r[1] * G[1], r[2] * G[1]};
    b[0] = -fma(r[0], g[0], G[0]), b[1] = -r[0] * g[1], b[2] = -r[0] * g[2];
    b[3] = -fma(r[1], g[1], G[0]), b[4] = -r[1] * g[2], b[5] = -fma(r[2], g[2], G[0]);
  }
  const int at[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double v = b[at[c][d]];
      B[(3 * (size_t)i + c) * N3 + 3 * (size_t)j + d] = zij ? 0.0 : v;
      if (i != j) B[(3 * (size_t)j + c) * N3 + 3 * (size_t)i + d] = zji ? 0.0 : v;
    }
}

// Component c of alpha^-1 (or alpha) times three values: the six upper entries.
__device__ __forceinline__ double sym_row(const double* __restrict__ a, int c, double x, double y,
                                          double z, double s) {
  const double ax = a[c], ay = c == 0 ? a[1] : c == 1 ? a[3] : a[4],
               az = c == 0 ? a[2] : c == 1 ? a[4] : a[5];
  // the diagonal entry last
  if (c == 0) return fma(ax, x, fma(ay, y, fma(az, z, s)));
  if (c == 1) return fma(ay, y, fma(ax, x, fma(az, z, s)));
  return fma(az, z, fma(ay, y, fma(ax, x, s)));
}

// out = B v, block per site; part (may be null): v . out of each site.  26 warps
// an SM at 999 sites keep enough of the matrix in flight.  flags: nothing to do
// once flags[0] is set (null: none).
__global__ void __launch_bounds__(DENSE_BLOCK)
      k_dense_apply(int n, const double* __restrict__ T, const double* __restrict__ ainv6,
                    const double* __restrict__ v, double* __restrict__ out, double* __restrict__ part,
                    const int* __restrict__ flags) {
  __shared__ double s_a[3][DENSE_BLOCK / 32];
  if (flags && flags[0]) return;
  const int i = blockIdx.x, N = 3 * n;
  const double* r = T + 3 * (size_t)i * N;
  double a[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int k = threadIdx.x; k < N; k += DENSE_BLOCK) {
    const double x = v[k];
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = fma(r[(size_t)c * N + k], x, a[c]);
  }
  // lanes 0-7: the warp's sum of a[0], 16-23 of a[1], 8-15 of a[2] (six additions, not 15)
  const bool up = threadIdx.x & 16, mid = threadIdx.x & 8;
  double t = (up ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, up ? a[0] : a[1], 16);
  a[2] += __shfl_xor_sync(0xffffffffu, a[2], 16);
  t = (mid ? a[2] : t) + __shfl_xor_sync(0xffffffffu, mid ? t : a[2], 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 7) == 0 && !(up && mid)) s_a[mid ? 2 : up ? 1 : 0][threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x < 3) {
    const int c    = threadIdx.x;
    const double* x = v + 3 * i;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < DENSE_BLOCK / 32; ++w) s += s_a[c][w];
    s              = sym_row(ainv6 + 6 * (size_t)i, c, x[0], x[1], x[2], s);
    out[3 * i + c] = s;
    const double d = x[c] * s;
    const double e = d + __shfl_sync(0x7u, d, 1) + __shfl_sync(0x7u, d, 2);
    if (part && c == 0) part[i] = e;
  }
}

// The warp's sums of u and v: of u in lanes 0-15, of v in lanes 16-31 (six
// additions a lane instead of ten: a quarter of an SM takes 64 clocks over each).
__device__ __forceinline__ double warp_sum2(double u, double v) {
  const bool hi = threadIdx.x & 16;
  double s      = (hi ? v : u) + __shfl_xor_sync(0xffffffffu, hi ? u : v, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The vector part of one CG iteration after B p (k_cg_update and k_cg_dir in
// one launch), by one cluster: p.Ap from the sites' values, x, r, z, the two
// dots through distributed shared memory, then p.  host_flags: pinned copy of
// flags[0..1].  999 sites: 11 us, a chain of some 70 FP64 instructions at 64
// clocks each and two cluster barriers; k_cg_update took 20 us with the direction
// in its last block, 8 and a further launch without.
__global__ void __cluster_dims__(STEP_CLUSTER) __launch_bounds__(STEP_BLOCK)
      k_dense_step(int n, const double* __restrict__ part, const double* __restrict__ Ap,
                   const double* __restrict__ a6, double* __restrict__ x, double* __restrict__ r,
                   double* __restrict__ p, double* scal, int* flags, double* __restrict__ hist,
                   double thresh, int maxiter, int* host_flags) {
  __shared__ double s_pap[STEP_BLOCK / 32], s_sum[2][STEP_BLOCK / 32];
  coop::cluster_group cl = coop::this_cluster();
  if (flags[0]) return;  // (every block reads it before the first cluster barrier)
  const int i     = blockIdx.x * STEP_BLOCK + threadIdx.x;
  const int lane  = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double rz = scal[S_RZ];
  const int it    = flags[1];
  double pv       = 0.0;
  for (int k = threadIdx.x; k < n; k += STEP_BLOCK) pv += part[k];
  pv = warp_sum(pv);
  if (lane == 0) s_pap[warp] = pv;
  __syncthreads();
  pv = (s_pap[0] + s_pap[1]) + (s_pap[2] + s_pap[3]);
  const double a = rz / pv;
  double v[2]    = {0.0, 0.0}, z[3], pc[3];
  if (i < n) {
    double rv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int k = 3 * i + c;
      pc[c]       = p[k];
      x[k]        = fma(a, pc[c], x[k]);
      rv[c]       = fma(-a, Ap[k], r[k]);
      r[k]        = rv[c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      z[c] = sym_row(a6 + 6 * (size_t)i, c, rv[0], rv[1], rv[2], 0.0);
      v[0] = fma(rv[c], rv[c], v[0]);
      v[1] = fma(rv[c], z[c], v[1]);
    }
  }
  v[0] = warp_sum2(v[0], v[1]);
  if ((lane & 15) == 0) s_sum[lane >> 4][warp] = v[0];
  cl.sync();
  // the cluster's 32 warps' values, one a lane
  const double* q  = cl.map_shared_rank(&s_sum[0][0], lane / (STEP_BLOCK / 32));
  const double s2  = warp_sum2(q[lane % (STEP_BLOCK / 32)], q[STEP_BLOCK / 32 + lane % (STEP_BLOCK / 32)]);
  const double rz1 = __shfl_sync(0xffffffffu, s2, 16);
  const double bt  = rz1 / rz;
  if (i < n)
#pragma unroll
    for (int c = 0; c < 3; ++c) p[3 * i + c] = fma(bt, pc[c], z[c]);
  if (i == 0) {
    const double rn = sqrt(s2);
    const int done  = rn < thresh ? 1 : it + 1 >= maxiter ? 2 : 0;
    hist[it]        = rn;
    scal[S_RNORM]   = rn;
    scal[S_RZOLD] = rz, scal[S_RZ] = rz1, scal[S_BETA] = bt;
    flags[1] = it + 1, flags[0] = done;
    host_flags[1] = it + 1, host_flags[0] = done;
  }
  cl.sync();  // the others' shared memory stays until everyone has read it
}

// The Jacobi-preconditioned CG of InducedMoments::compute
// (src/core/electric_fields.cc:191-239) by one block with the matrix in shared
// memory (column-major), L threads per row: one launch and one
// synchronisation per solve instead of four launches per iteration.  A quarter
// of an SM takes 64 clocks over an FP64 instruction of a warp, whatever its
// lanes do: L is chosen for four warps, and every scalar counts.
// 18 sites, 15 iterations: 55 us (97 us with eight threads per row, 74 us with
// one); a solve through the C call takes 66 us, 562 us with the launches.  rhs,
// guess and mu may be host memory the device can address; hist receives r.r per
// iteration.
template <int L>
__global__ void __launch_bounds__(SMALL_THREADS)
      k_solve_small(int n, const double* __restrict__ Tg, const double* __restrict__ ainv6,
                    const double* __restrict__ alpha6, const double* __restrict__ rhs,
                    const double* __restrict__ guess, int make_guess, double thresh2, int maxiter,
                    double* __restrict__ mu, double* __restrict__ hist, double* __restrict__ scal,
                    int* __restrict__ flags) {
  extern __shared__ __align__(16) double s_T[];
  const int N = 3 * n, nw = blockDim.x >> 5;
  double* s_v = s_T + (size_t)N * N;  // the vector the matrix is applied to
  double* s_r = s_v + N;
  __shared__ double sh1[SMALL_THREADS / 32], sh2[2][SMALL_THREADS / 32];
  const int k    = threadIdx.x / L, l = threadIdx.x % L;
  const bool row = k < N, own = row && l == 0;
#pragma unroll 8
  for (int q = threadIdx.x; q < N * N; q += blockDim.x) s_T[(q % N) * N + q / N] = Tg[q];
  const int i = row ? k / 3 : 0, c = row ? k - 3 * i : 0;
  double al[6], ai[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) al[q] = alpha6[6 * i + q], ai[q] = ainv6[6 * i + q];
  auto sym = [&](const double* a, const double* x, double s) {
    return sym_row(a, c, x[3 * i], x[3 * i + 1], x[3 * i + 2], s);
  };
  // (every lane of a row holds the row's values)
  auto apply = [&]() {  // row k of B s_v
    __syncthreads();
    double a = 0.0, b = 0.0, d = 0.0;
    if (row) {
      int q = l;
      for (; q + 2 * L < N; q += 3 * L) {
        a = fma(s_T[q * N + k], s_v[q], a);
        b = fma(s_T[(q + L) * N + k], s_v[q + L], b);
        d = fma(s_T[(q + 2 * L) * N + k], s_v[q + 2 * L], d);
      }
      if (q < N) a = fma(s_T[q * N + k], s_v[q], a);
      if (q + L < N) b = fma(s_T[(q + L) * N + k], s_v[q + L], b);
    }
    a += b + d;
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return row ? sym(ai, s_v, a) : 0.0;
  };
  auto precond = [&](double r) {  // row k of alpha r (s_r: a barrier follows each use)
    if (own) s_r[k] = r;
    __syncthreads();
    return row ? sym(al, s_r, 0.0) : 0.0;
  };
  auto sum1 = [&](double v) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh1[threadIdx.x >> 5] = v;
    __syncthreads();
    v = sh1[0];
    for (int w = 1; w < nw; ++w) v += sh1[w];
    return v;
  };
  auto sum2 = [&](double& u, double& v) {
    u = warp_sum2(u, v);
    if ((threadIdx.x & 15) == 0) sh2[(threadIdx.x >> 4) & 1][threadIdx.x >> 5] = u;
    __syncthreads();
    u = sh2[0][0], v = sh2[1][0];
    for (int w = 1; w < nw; ++w) u += sh2[0][w], v += sh2[1][w];
  };
  const double F = row ? rhs[k] : 0.0;
  double x = 0.0, r = F;
  if (make_guess)
    x = precond(F);
  else if (guess && row)
    x = guess[k];
  if (make_guess || guess) {
    if (own) s_v[k] = x;
    r = F - apply();
  }
  double z = precond(r), p = z;
  double rz = own ? r * z : 0.0, rr = own ? r * r : 0.0;
  sum2(rz, rr);
  int it = 0, done = 0;
  while (!done && it < maxiter) {
    // (s_v: every thread has passed a barrier since it last read it)
    if (own) s_v[k] = p;
    const double Ap = apply();
    const double a  = rz / sum1(own ? p * Ap : 0.0);
    x               = fma(a, p, x);
    r               = fma(-a, Ap, r);
    z               = precond(r);
    double rz1      = own ? r * z : 0.0;
    rr              = own ? r * r : 0.0;
    sum2(rz1, rr);
    if (threadIdx.x == 0) hist[it] = rr;
    ++it;
    done = rr < thresh2 ? 1 : it >= maxiter ? 2 : 0;
    p    = fma(rz1 / rz, p, z);
    rz   = rz1;
  }
  if (own) mu[k] = x;
  if (threadIdx.x == 0) scal[S_RNORM] = rr, flags[0] = done, flags[1] = it;
}

static size_t small_smem(int n) { return sizeof(double) * (3 * (size_t)n) * (3 * (size_t)n + 2); }

// Bytes of all systems' matrices in this process.
static std::atomic<size_t> s_dense_bytes{0};

bool System::dense_operator() const {
  return !geo.fmm && opt.precision == CPPE_GPU_FP64 && n <= DENSE_MAX && dense != DENSE_NONE;
}

// Builds the matrix on first use; false (for good) where the matrices of other
// systems leave no room for it or the device has none: the pair kernels then serve
// this system, as they serve larger ones.
bool System::dense_build() {
  if (dense != DENSE_UNTRIED) return dense == DENSE_BUILT;
  const size_t N3 = 3 * (size_t)n, bytes = N3 * N3 * sizeof(double);
  dense = DENSE_NONE;
  if (s_dense_bytes.fetch_add(bytes) + bytes > DENSE_POOL) {
    s_dense_bytes -= bytes;
    return false;
  }
  dense_bytes = bytes;
  try {
    Tmat.alloc(N3 * N3);
  } catch (const Failure&) {
    cudaGetLastError();  // (out of memory is not sticky)
    dense_release();
    return false;
  }
  const long pairs = (long)n * (n + 1) / 2;
  k_dense_build<<<(unsigned)((pairs + 127) / 128), 128, 0, stream>>>(
        n, geo.pos64.p, geo.corr_ptr.p, geo.corr_idx.p, opt.damp != 0, opt.damping_factor, Tmat.p);
  CG_LAUNCH();
  dense = DENSE_BUILT;
  return true;
}

void System::dense_release() {
  Tmat.release();
  s_dense_bytes -= dense_bytes;
  dense_bytes = 0;
}

void System::dense_apply(const double* in, double* out, bool iteration) {
  k_dense_apply<<<n, DENSE_BLOCK, 0, stream>>>(n, Tmat.p, ainv64.p, in, out,
                                               iteration ? partials.p : nullptr,
                                               iteration ? flags.p : nullptr);
  CG_LAUNCH();
}

// One CG iteration; host_flags follows flags.
void System::dense_iteration() {
  dense_apply(p.p, Ap.p, true);
  k_dense_step<<<STEP_CLUSTER, STEP_BLOCK, 0, stream>>>(n, partials.p, Ap.p, alpha64.p, x.p, r.p,
                                                        p.p, scal.p, flags.p, hist.p,
                                                        opt.induced_thresh, opt.maxiter, h_flags);
  CG_LAUNCH();
}

bool System::small_solver() {
  // (its stopping rule compares squares; with a limit of more iterations than it
  // could take in some milliseconds, the loop of launches, which the host can leave)
  return dense_operator() && n <= SMALL_MAX && opt.maxiter <= SMALL_MAXITER && !model &&
         opt.induced_thresh > 1e-140 && dense_build();
}

int System::solve_small(const double* rhs, const double* guess, int make_guess, double* mu,
                        int* iters, double* hist_out, int hist_cap) {
  if (!h_hist) CG_CUDA(cudaMallocHost(&h_hist, sizeof(double) * (std::max(1, opt.maxiter) + 64)));
  if (!small_ready) {
    CG_CUDA(cudaFuncSetAttribute(k_solve_small<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)small_smem(SMALL_MAX)));
    small_ready = true;
  }
  // (lanes of an idle quarter of the SM cost nothing, more than four warps do)
  const int lanes = 12 * n <= 128 ? 4 : 6 * n <= 128 ? 2 : 1;
  auto kern       = lanes == 4 ? k_solve_small<4> : lanes == 2 ? k_solve_small<2> : k_solve_small<1>;
  kern<<<1, (3 * n * lanes + 31) / 32 * 32, small_smem(n), stream>>>(
        n, Tmat.p, ainv64.p, alpha64.p, rhs, guess, make_guess,
        opt.induced_thresh * opt.induced_thresh, opt.maxiter, mu, h_hist, h_scal, h_flags);
  CG_LAUNCH();
  CG_CUDA(cudaStreamSynchronize(stream));
  last              = SolveStats();
  last.iterations   = h_flags[1];
  last.final_rnorm  = std::sqrt(h_scal[S_RNORM]);
  last.fp64_applies = h_flags[1] + (make_guess || guess ? 1 : 0);
  if (iters) *iters = h_flags[1];
  if (hist_out)
    for (int k = 0; k < std::min(h_flags[1], hist_cap); ++k) hist_out[k] = std::sqrt(h_hist[k]);
  return h_flags[0] == 1 ? CPPE_GPU_OK : CPPE_GPU_NOT_CONVERGED;
}

}  // namespace cg
