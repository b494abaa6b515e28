// MLP kernels: tiled SIMT GEMMs with bias, GELU and split-K epilogues, the output
// layer with the loss of the learned guess + preconditioner correction, Adam.
#include <cmath>
#include <random>

#include "mlp.h"

namespace cg {

constexpr int GT = 64, GK = 16, GEMM_THREADS = 128;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678f)) + z * __expf(-0.5f * z * z) * 0.39894228f;
}

// C = op(A) op(B): A(m,k) = TA ? A[k lda + m] : A[m lda + k],
//                  B(k,n) = TB ? B[n ldb + k] : B[k ldb + n].
// Block: 64 x 64 outputs, 128 threads with 8 x 4 each; 16384 x 128 x 128 takes
// 22 us, 7 us of them multiply-adds, the rest mostly the epilogue, the start and 3.4
// blocks an SM that run as 4.  The next 16 k's loads are in flight while the last 16 are
// multiplied.  K is a multiple of 4 if A is not transposed, N, lda and ldb are
// multiples of 4, A and B 16-byte aligned.  FP32 throughout.
enum Epilogue {
  EPI_BIAS,       // C = A B + bias
  EPI_GELU,       // C = A B + bias, C2 = gelu(C)
  EPI_GELU_BACK,  // C = A B * gelu'(Z)
  EPI_PARTIAL     // blockIdx.z's k's only, into part z of C (ld_part apart), with the
                  // sums of A over k in C2: a weight's and its bias' gradient
};
// (x - mean) * inv_std over the columns of a raw operand
struct Norm {
  const float *mean, *inv_std;
  __device__ __forceinline__ float4 operator()(float4 x, int c) const {
    const float4 m = *reinterpret_cast<const float4*>(mean + c);
    const float4 d = *reinterpret_cast<const float4*>(inv_std + c);
    return make_float4((x.x - m.x) * d.x, (x.y - m.y) * d.y, (x.z - m.z) * d.z,
                       (x.w - m.w) * d.w);
  }
};
// NORM: A (B in EPI_PARTIAL) is the raw input.
template <bool TA, bool TB, int EPI, bool NORM>
__global__ void __launch_bounds__(GEMM_THREADS, 4)
      k_gemm(int M, int N, int K, const float* __restrict__ A, int lda,
             const float* __restrict__ B, int ldb, float* __restrict__ C, float* __restrict__ C2,
             const float* __restrict__ bias, const float* __restrict__ Z, Norm norm, int kchunk,
             int ld_part) {
  __shared__ __align__(16) float As[2][GK][GT + 4];
  __shared__ __align__(16) float Bs[2][GK][GT + 4];
  constexpr bool PART = EPI == EPI_PARTIAL;
  const int m0 = blockIdx.y * GT, n0 = blockIdx.x * GT;
  const int kbeg = PART ? blockIdx.z * kchunk : 0, kend = PART ? min(K, kbeg + kchunk) : K;
  // a warp's outputs are 2 x 16 rows by 32 columns: its reads of a column of As or a
  // row of Bs are one wavefront each
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = (lane & 7) + 8 * (warp & 1), ty = (lane >> 3) + 4 * (warp >> 1);
  // this thread's two groups of four values of a tile: along k, or across it
  auto load = [&](bool across, bool nrm, const float* P, int ld, int r0, int R, int k0,
                  float4 (&v)[2]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = threadIdx.x + GEMM_THREADS * q;
      const int r = r0 + (across ? (e & 15) * 4 : e >> 2);
      const int k = k0 + (across ? e >> 4 : (e & 3) * 4);
      v[q]        = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < R && k < kend) {
        v[q] = *reinterpret_cast<const float4*>(P + (across ? (size_t)k * ld + r
                                                            : (size_t)r * ld + k));
        if (nrm) v[q] = norm(v[q], across ? r : k);
      }
    }
  };
  auto store = [&](bool across, float (*S)[GT + 4], const float4 (&v)[2]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = threadIdx.x + GEMM_THREADS * q;
      if (across) {
        *reinterpret_cast<float4*>(&S[e >> 4][(e & 15) * 4]) = v[q];
      } else {
        const int k = (e & 3) * 4, r = e >> 2;
        S[k][r] = v[q].x, S[k + 1][r] = v[q].y, S[k + 2][r] = v[q].z, S[k + 3][r] = v[q].w;
      }
    }
  };
  float acc[8][4], asum[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    asum[i] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  }
  float4 a4[2], b4[2];
  load(TA, NORM && !PART, A, lda, m0, M, kbeg, a4), load(!TB, NORM && PART, B, ldb, n0, N, kbeg, b4);
  store(TA, As[0], a4), store(!TB, Bs[0], b4);
  int cur = 0;
  for (int k0 = kbeg; k0 < kend; k0 += GK, cur ^= 1) {
    __syncthreads();
    const bool more = k0 + GK < kend;
    if (more) {
      load(TA, NORM && !PART, A, lda, m0, M, k0 + GK, a4);
      load(!TB, NORM && PART, B, ldb, n0, N, k0 + GK, b4);
    }
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      const float4 av = *reinterpret_cast<const float4*>(&As[cur][kk][ty * 4]);
      const float4 aw = *reinterpret_cast<const float4*>(&As[cur][kk][GT / 2 + ty * 4]);
      const float4 bv = *reinterpret_cast<const float4*>(&Bs[cur][kk][tx * 4]);
      const float a[8] = {av.x, av.y, av.z, av.w, aw.x, aw.y, aw.z, aw.w};
      const float b[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      if (PART && blockIdx.x == 0)
#pragma unroll
        for (int i = 0; i < 8; ++i) asum[i] += a[i];
    }
    // (the other buffer's readers passed the barrier above)
    if (more) store(TA, As[cur ^ 1], a4), store(!TB, Bs[cur ^ 1], b4);
  }
  const int n = n0 + tx * 4;
  if (n >= N) return;
  if (PART) C += (size_t)blockIdx.z * ld_part, C2 += (size_t)blockIdx.z * ld_part;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + (i < 4 ? 0 : GT / 2) + ty * 4 + (i & 3);
    if (m >= M) continue;
    const size_t at = (size_t)m * N + n;
    if (EPI == EPI_BIAS || EPI == EPI_GELU)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += bias[n + j];
    if (EPI == EPI_GELU_BACK) {
      const float4 z = *reinterpret_cast<const float4*>(Z + at);
      acc[i][0] *= gelu_grad(z.x), acc[i][1] *= gelu_grad(z.y);
      acc[i][2] *= gelu_grad(z.z), acc[i][3] *= gelu_grad(z.w);
    }
    if (PART && n == 0) C2[m] = asum[i];
    *reinterpret_cast<float4*>(C + at) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    if (EPI == EPI_GELU)
      *reinterpret_cast<float4*>(C2 + at) =
            make_float4(gelu(acc[i][0]), gelu(acc[i][1]), gelu(acc[i][2]), gelu(acc[i][3]));
  }
}

static dim3 gemm_grid(int M, int N, int splits) {
  return dim3((N + GT - 1) / GT, (M + GT - 1) / GT, splits);
}

// The output layer, forward and back, the loss (see oracle/mlp_oracle.py for its
// definition) and the gradient with respect to the second layer's
// pre-activations, in one pass over H2 and Z2: a warp per row, four of the 128
// columns a lane.  Block z takes the rows of part z and leaves its share of
// dW3 and db3 there.  15 us for 16384 rows; as GEMMs, 4 wide, 18 us
// forward, 107 + 35 us for dW3 and db3, 33 us for dZ2.  The loss terms, FP64, are
// left to four warps per 128 rows: an SM issues two FP64 lanes a clock.
constexpr int HEAD_WARPS = 16, HEAD_ROWS = 128;
__global__ void __launch_bounds__(32 * HEAD_WARPS)
      k_head(int B, int rows_per, const float* __restrict__ H2, const float* __restrict__ Z2,
             const float* __restrict__ W3, const float* __restrict__ b3,
             const float* __restrict__ T, float lam, float* __restrict__ dZ2,
             float* __restrict__ part, int ld_part, double* __restrict__ loss_part) {
  constexpr int H = Mlp::H, OUT = Mlp::OUT;
  static_assert(H == 128 && OUT == 4, "a float4 of a row per lane, four outputs");
  __shared__ __align__(16) float s_g[HEAD_WARPS][OUT * H];
  __shared__ float s_b[HEAD_WARPS][OUT];
  __shared__ float s_d[HEAD_ROWS][8];
  __shared__ double s_l[HEAD_ROWS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.x * rows_per, r1 = min(B, r0 + rows_per);
  float w[OUT][4], gw[OUT][4], gb[OUT];
#pragma unroll
  for (int o = 0; o < OUT; ++o) {
    const float4 v = *reinterpret_cast<const float4*>(W3 + o * H + 4 * lane);
    w[o][0] = v.x, w[o][1] = v.y, w[o][2] = v.z, w[o][3] = v.w;
    gw[o][0] = gw[o][1] = gw[o][2] = gw[o][3] = gb[o] = 0.f;
  }
  const float bias[OUT] = {b3[0], b3[1], b3[2], b3[3]};
  const float invB      = 1.f / (float)B;
  double l              = 0.0;
  for (int rb = r0; rb < r1; rb += HEAD_ROWS) {
    const int re = min(r1, rb + HEAD_ROWS);
#pragma unroll 2
    for (int r = rb + warp; r < re; r += HEAD_WARPS) {
      const float4 hv  = *reinterpret_cast<const float4*>(H2 + (size_t)r * H + 4 * lane);
      const float4 zv  = *reinterpret_cast<const float4*>(Z2 + (size_t)r * H + 4 * lane);
      float t[Mlp::TROW];
#pragma unroll
      for (int q = 0; q < Mlp::TROW / 4; ++q)
        *reinterpret_cast<float4*>(t + 4 * q) =
              *reinterpret_cast<const float4*>(T + (size_t)r * Mlp::TROW + 4 * q);
      const float h[4] = {hv.x, hv.y, hv.z, hv.w};
      float y[OUT];
#pragma unroll
      for (int o = 0; o < OUT; ++o) {
        y[o] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) y[o] = fmaf(h[j], w[o][j], y[o]);
      }
      // output o's sum in the lanes with bits 3 and 4 = o
      const bool up = lane & 16, mid = lane & 8;
      const float y0 = (up ? y[2] : y[0]) + __shfl_xor_sync(0xffffffffu, up ? y[0] : y[2], 16);
      const float y1 = (up ? y[3] : y[1]) + __shfl_xor_sync(0xffffffffu, up ? y[1] : y[3], 16);
      float ys       = (mid ? y1 : y0) + __shfl_xor_sync(0xffffffffu, mid ? y0 : y1, 8);
#pragma unroll
      for (int q = 4; q > 0; q >>= 1) ys += __shfl_xor_sync(0xffffffffu, ys, q);
#pragma unroll
      for (int o = 0; o < OUT; ++o) y[o] = __shfl_sync(0xffffffffu, ys, 8 * o) + bias[o];
      float dg[3], dp[3], g[4] = {0.f, 0.f, 0.f, 0.f};
      const float s = t[21], u = t[22];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        dg[c] = y[0] * t[c] + y[1] * t[3 + c] + y[2] * t[6 + c] - t[9 + c];
        dp[c] = t[12 + c] + y[3] * t[15 + c] - t[18 + c];
        g[0] += dg[c] * t[c];
        g[1] += dg[c] * t[3 + c];
        g[2] += dg[c] * t[6 + c];
        g[3] += dp[c] * t[15 + c];
      }
      if (lane == 0) {
        float* d = s_d[r - rb];
        d[0] = dg[0], d[1] = dg[1], d[2] = dg[2], d[3] = s;
        d[4] = dp[0], d[5] = dp[1], d[6] = dp[2], d[7] = u;
      }
      // one of the four quotients a lane
      const float go = up ? (mid ? 2.f * lam * g[3] : 2.f * g[2]) : 2.f * (mid ? g[1] : g[0]);
      const float dq = go / (up && mid ? u : s) * invB;
      float dy[OUT];
#pragma unroll
      for (int o = 0; o < OUT; ++o) dy[o] = __shfl_sync(0xffffffffu, dq, 8 * o);
      float dh[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int o = 0; o < OUT; ++o) {
        gb[o] += dy[o];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dh[j]    = fmaf(dy[o], w[o][j], dh[j]);
          gw[o][j] = fmaf(dy[o], h[j], gw[o][j]);
        }
      }
      *reinterpret_cast<float4*>(dZ2 + (size_t)r * H + 4 * lane) =
            make_float4(dh[0] * gelu_grad(zv.x), dh[1] * gelu_grad(zv.y),
                        dh[2] * gelu_grad(zv.z), dh[3] * gelu_grad(zv.w));
    }
    __syncthreads();
    if (threadIdx.x < re - rb) {
      const float* d = s_d[threadIdx.x];
      double lg = 0.0, lp = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        lg += (double)d[c] * d[c];
        lp += (double)d[4 + c] * d[4 + c];
      }
      l += (lg / d[3] + lam * lp / d[7]) / B;
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 0; o < OUT; ++o) {
    *reinterpret_cast<float4*>(&s_g[warp][o * H + 4 * lane]) =
          make_float4(gw[o][0], gw[o][1], gw[o][2], gw[o][3]);
    if (lane == 0) s_b[warp][o] = gb[o];
  }
  if (warp < HEAD_ROWS / 32) {
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) l += __shfl_xor_sync(0xffffffffu, l, q);
    if (lane == 0) s_l[warp] = l;
  }
  __syncthreads();
  if (threadIdx.x == 0) loss_part[blockIdx.x] = (s_l[0] + s_l[1]) + (s_l[2] + s_l[3]);
  part += (size_t)blockIdx.x * ld_part;
  for (int k = threadIdx.x; k < OUT * H + OUT; k += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < HEAD_WARPS; ++q) v += k < OUT * H ? s_g[q][k] : s_b[q][k - OUT * H];
    part[k] = v;
  }
}

// The sum of the parts of every parameter's gradient (thread g of a parameter's
// eight takes parts g, g + 8, ...; one after the other took 12 us and rounded
// more often) and of the loss, which goes to pinned memory.
constexpr int SUM_LANES = 8;
__global__ void __launch_bounds__(32 * SUM_LANES)
      k_sum_parts(int n, int parts, const float* __restrict__ part, float* __restrict__ out,
                  const double* __restrict__ loss_part, double* __restrict__ loss) {
  __shared__ float s_p[SUM_LANES][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, t = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (t < n)
#pragma unroll 8
    for (int z = g; z < parts; z += SUM_LANES) s += part[(size_t)z * n + t];
  s_p[g][lane] = s;
  __syncthreads();
  if (g == 0 && t < n) {
    float v[SUM_LANES];
#pragma unroll
    for (int q = 0; q < SUM_LANES; ++q) v[q] = s_p[q][lane];
    out[t] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  if (blockIdx.x == 0 && g == 1) {
    double l = 0.0;
    for (int z = lane; z < parts; z += 32) l += loss_part[z];
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) l += __shfl_xor_sync(0xffffffffu, l, q);
    if (lane == 0) *loss = l;
  }
}

__global__ void k_adam(int n, float* __restrict__ w, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float gt = g[t];
  const float mt = b1 * m[t] + (1.f - b1) * gt;
  const float vt = b2 * v[t] + (1.f - b2) * gt * gt;
  m[t] = mt, v[t] = vt;
  w[t] -= lr * (mt / c1) / (sqrtf(vt / c2) + eps);
}

Mlp::~Mlp() {
  if (stream) {
    cudaSetDevice(device);
    cudaStreamSynchronize(stream);
    cudaStreamDestroy(stream);
  }
  if (h_loss) cudaFreeHost(h_loss);
}

void Mlp::init(int dev, unsigned seed) {
  device = dev;
  CG_CUDA(cudaSetDevice(device));
  CG_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  std::mt19937 rng(seed);
  std::vector<float> p(NPARAM, 0.f);
  auto fill = [&](int off, int cnt, float scale) {
    std::uniform_real_distribution<float> u(-scale, scale);
    for (int k = 0; k < cnt; ++k) p[off + k] = u(rng);
  };
  fill(0, NW1, 1.f / std::sqrt((float)IN));
  fill(NW1 + NB1, NW2, 1.f / std::sqrt((float)H));
  fill(NW1 + NB1 + NW2 + NB2, NW3, 0.01f / std::sqrt((float)H));
  // output bias: start at the three-term series mu = v1 + v2 + v3 and no correction
  float* b3h = &p[NW1 + NB1 + NW2 + NB2 + NW3];
  b3h[0] = 1.f, b3h[1] = 1.f, b3h[2] = 1.f, b3h[3] = 0.f;
  params.upload(p, stream);
  grads.alloc(NPARAM);
  adam_m.alloc(NPARAM);
  adam_v.alloc(NPARAM);
  adam_m.zero(stream);
  adam_v.zero(stream);
  std::vector<float> mean(IN, 0.f), istd(IN, 1.f);
  feat_mean.upload(mean, stream);
  feat_inv_std.upload(istd, stream);
  CG_CUDA(cudaMallocHost(&h_loss, sizeof(double)));
  tc_err.alloc(1);
  tc_err.zero(stream);
  step = 0;
  CG_CUDA(cudaStreamSynchronize(stream));
}

void Mlp::reserve(int rows) {
  if (rows <= cap) return;
  cap = rows;
  Z1.alloc((size_t)rows * H), H1.alloc((size_t)rows * H);
  Z2.alloc((size_t)rows * H), H2.alloc((size_t)rows * H);
  dZ1.alloc((size_t)rows * H), dZ2.alloc((size_t)rows * H);
  part.alloc((size_t)MAX_PARTS * NPARAM);
  loss_part.alloc(MAX_PARTS);
}

void Mlp::upload(DBuf<float>& d, const float* h, size_t count) {
  if (d.n < count) d.alloc(count);
  CG_CUDA(cudaMemcpyAsync(d.p, h, count * sizeof(float), cudaMemcpyHostToDevice, stream));
}

// Inference on the tensor cores (mlp_tc.cu); tc_err reports a timed-out wait.
void Mlp::infer(int rows, const float* raw, float* Y_out, cudaStream_t s) {
  if (rows <= 0) return;
  tc_err.zero(s);
  mlp_infer_tc(device, rows, raw, params.p, feat_mean.p, feat_inv_std.p, Y_out, tc_err.p, s);
}

// The two hidden layers of the raw rows, which are normalised as they are read.
void Mlp::hidden(int rows, const float* raw, cudaStream_t s) {
  reserve(rows);
  const Norm norm{feat_mean.p, feat_inv_std.p};
  k_gemm<false, true, EPI_GELU, true><<<gemm_grid(rows, H, 1), GEMM_THREADS, 0, s>>>(
        rows, H, IN, raw, IN, W1(), IN, Z1.p, H1.p, b1(), nullptr, norm, 0, 0);
  CG_LAUNCH();
  k_gemm<false, true, EPI_GELU, false><<<gemm_grid(rows, H, 1), GEMM_THREADS, 0, s>>>(
        rows, H, H, H1.p, H, W2(), H, Z2.p, H2.p, b2(), nullptr, norm, 0, 0);
  CG_LAUNCH();
}

void Mlp::forward(int rows, const float* raw, float* Y_out, cudaStream_t s) {
  hidden(rows, raw, s);
  k_gemm<false, true, EPI_BIAS, false><<<gemm_grid(rows, OUT, 1), GEMM_THREADS, 0, s>>>(
        rows, OUT, H, H2.p, H, W3(), H, Y_out, nullptr, b3(), nullptr, Norm(), 0, 0);
  CG_LAUNCH();
}

// The gradients are sums over the rows: up to MAX_PARTS parts of whole GEMM steps,
// at least 32 rows each, fill the chip (a 128 x 128 weight is four tiles).  16384
// rows: 116 us in seven kernels, 640 us in 22 before (three 107 us weight gradients on
// 64 blocks, 150 us of bias sums); the gradients' error is 2.5 times smaller for the
// shorter sums.
double Mlp::loss_grad(int rows, const float* raw, const float* targets, float lam) {
  CG_CUDA(cudaSetDevice(device));
  cudaStream_t s = stream;
  hidden(rows, raw, s);
  const int want  = std::max(1, std::min(MAX_PARTS, rows / 32));
  const int chunk = ((rows + want - 1) / want + GK - 1) / GK * GK;
  const int parts = (rows + chunk - 1) / chunk;
  float* gW1 = part.p;  // (of the first part; the others NPARAM apart)
  float* gb1 = gW1 + NW1;
  float* gW2 = gb1 + NB1;
  float* gb2 = gW2 + NW2;
  float* gW3 = gb2 + NB2;
  const Norm norm{feat_mean.p, feat_inv_std.p};
  k_head<<<parts, 32 * HEAD_WARPS, 0, s>>>(rows, chunk, H2.p, Z2.p, W3(), b3(), targets, lam,
                                           dZ2.p, gW3, NPARAM, loss_part.p);
  CG_LAUNCH();
  // layer 2: dW2 = dZ2^T H1, db2, dZ1 = dZ2 W2 gelu'(Z1)
  k_gemm<true, false, EPI_PARTIAL, false><<<gemm_grid(H, H, parts), GEMM_THREADS, 0, s>>>(
        H, H, rows, dZ2.p, H, H1.p, H, gW2, gb2, nullptr, nullptr, norm, chunk, NPARAM);
  CG_LAUNCH();
  k_gemm<false, false, EPI_GELU_BACK, false><<<gemm_grid(rows, H, 1), GEMM_THREADS, 0, s>>>(
        rows, H, H, dZ2.p, H, W2(), H, dZ1.p, nullptr, nullptr, Z1.p, norm, 0, 0);
  CG_LAUNCH();
  // layer 1: dW1 = dZ1^T X, db1
  k_gemm<true, false, EPI_PARTIAL, true><<<gemm_grid(H, IN, parts), GEMM_THREADS, 0, s>>>(
        H, IN, rows, dZ1.p, H, raw, IN, gW1, gb1, nullptr, nullptr, norm, chunk, NPARAM);
  CG_LAUNCH();
  k_sum_parts<<<(NPARAM + 31) / 32, 32 * SUM_LANES, 0, s>>>(NPARAM, parts, part.p, grads.p,
                                                            loss_part.p, h_loss);
  CG_LAUNCH();
  CG_CUDA(cudaStreamSynchronize(s));
  return *h_loss;
}

void Mlp::adam(float lr, float b1, float b2, float eps) {
  ++step;
  const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);
  k_adam<<<(NPARAM + 255) / 256, 256, 0, stream>>>(NPARAM, params.p, grads.p, adam_m.p, adam_v.p,
                                                   lr, b1, b2, eps, c1, c2);
  CG_LAUNCH();
}

}  // namespace cg
