// M2L with the expansion order fixed at compile time (the orders the
// benchmark configurations use; other orders take the table-driven k_m2l).
//
// Same operator as k_m2l (src/core/fmm/calculate.cc:186-203 with the
// field_m*.cc M2L kernels), organised for registers: each lane of a warp
// takes its own source cell of the target's interaction list, evaluates the
// straight-line translation generated by gen_m2l.py (derivative tensor and
// partial local expansion in registers, the source multipole streamed one
// coefficient at a time), and the lanes' partial expansions are added over the
// warp in a fixed order at the end (m2l_scatter).
//
// The translation works between harmonic-reduced coefficients (z-power 0 or 1,
// see gen_m2l.py): k_m2l_fold turns each cell's multipole into its reduced row
// before, k_lsum gives back the full local expansion after.  Measured (M2L
// phase with folding and per-cell sums, 300,000 sites order 6, 14.6 M
// translations; full coefficients -> reduced -> with the lanes' sums scattered
// and the recurrence's factors taken out):
//   FP32         1.54 -> 0.83 -> 0.61 ms
//   double-float 13.8 -> 7.8 -> 5.0 ms (also: source rows loaded an order ahead
//                two coefficients at a time, tensors copied row by row)
//   FP64         24.9 -> 14.9 -> 12.6 ms (bound by the FP64 pipe)
#pragma once

#include "dd.cuh"
#include "engine.h"

namespace cg {

// generated straight-line translations (function templates + an X-macro list)
#include "m2l_gen.cuh"

constexpr int nterms_c(int p) { return p < 0 ? 0 : (p + 1) * (p + 2) * (p + 3) / 6; }
// reduced coefficients (z-power 0 or 1) of orders 0..p
constexpr int nred(int p) { return p < 0 ? 0 : (p + 1) * (p + 1); }

// Derivative tensors of the distinct M2L vectors (Geometry::make_vectors),
// thread per vector, in T or in double-float.
#define CPPE_DEF_DTAB(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                                \
  template <typename T>                                                                     \
  __global__ void k_dtab_##NAME(int nvec, const double4_32a* __restrict__ vec,              \
                                T* __restrict__ D) {                                        \
    const int v = blockIdx.x * blockDim.x + threadIdx.x;                                    \
    if (v >= nvec) return;                                                                  \
    const double4_32a r = vec[v];                                                           \
    dtensor_##NAME<T>((T)r.x, (T)r.y, (T)r.z, D + (size_t)v * (NT));                        \
  }                                                                                         \
  template <int DD>                                                                         \
  __global__ void k_dtab_##NAME##_dd(int nvec, const double4_32a* __restrict__ vec,         \
                                     float2* __restrict__ D) {                              \
    const int v = blockIdx.x * blockDim.x + threadIdx.x;                                    \
    if (v >= nvec) return;                                                                  \
    const double4_32a r = vec[v];                                                           \
    ddv t[NT];                                                                              \
    dtensor_##NAME<ddv>(ddv(dd_from(r.x)), ddv(dd_from(r.y)), ddv(dd_from(r.z)), t);       \
    _Pragma("unroll") for (int j = 0; j < (NT); ++j)                                        \
          D[(size_t)v * (NT) + j] = make_float2(t[j].h, t[j].l);                            \
  }
CPPE_M2L_REDUCED(CPPE_DEF_DTAB)
#undef CPPE_DEF_DTAB

// Builds the tensor table of g's M2L vectors for order p into w (T, or
// double-float when dd) on first use; returns it, or null when g has no
// vector table or no fixed-order kernel serves (m, p).
template <bool DD, typename T>
const void* m2l_dtab(const Geometry& g, int m, int p, FieldWork<T>& w, cudaStream_t s) {
  const int nv = (int)g.h_vec.size();
  if (nv == 0) return nullptr;
  const void* out = nullptr;
#define CPPE_BUILD_DTAB(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                               \
  if (!out && m == MM && p == PP) {                                                          \
    const size_t cnt = (size_t)nv * (NT);                                                    \
    if constexpr (DD) {                                                                      \
      if constexpr (MM == 1) {                                                               \
        if (w.dtab_dd.n != cnt) {                                                            \
          w.dtab_dd.alloc(cnt);                                                              \
          k_dtab_##NAME##_dd<1><<<(nv + 63) / 64, 64, 0, s>>>(nv, g.vec.p, w.dtab_dd.p);     \
          CG_LAUNCH();                                                                       \
        }                                                                                    \
        out = w.dtab_dd.p;                                                                   \
      }                                                                                      \
    } else {                                                                                 \
      if (w.dtab.n != cnt) {                                                                 \
        w.dtab.alloc(cnt);                                                                   \
        k_dtab_##NAME<T><<<(nv + 63) / 64, 64, 0, s>>>(nv, g.vec.p, w.dtab.p);               \
        CG_LAUNCH();                                                                         \
      }                                                                                      \
      out = w.dtab.p;                                                                        \
    }                                                                                        \
  }
  CPPE_M2L_REDUCED(CPPE_BUILD_DTAB)
#undef CPPE_BUILD_DTAB
  return out;
}

// Reduced multipole rows Mr (stride m_stride(MS)) of every cell from the full
// ones (stride mstride); thread per (cell, reduced row).  To double-float
// pairs for the double-float translation (sums in T).
__device__ __forceinline__ void m2l_store(float& o, float v) { o = v; }
__device__ __forceinline__ void m2l_store(double& o, double v) { o = v; }
__device__ __forceinline__ void m2l_store(float2& o, double v) {
  const float h = (float)v;
  o             = make_float2(h, (float)(v - (double)h));
}
// Double-float rows: every order starts on a 16-byte boundary (2 o + 2 pairs
// for order o), so that the translation loads two coefficients at a time.
constexpr int m2l_dd_off(int m, int o) {
  int b = 0;
  for (int q = m; q < o; ++q) b += 2 * q + 2;
  return b;
}
template <typename O>
struct FoldRow {  // plain rows: stride and reduced coefficient of a position
  static constexpr int stride(int, int, int ms) { return m_stride(ms); }
  __host__ __device__ static constexpr int coef(int, int, int ms, int r) { return r < ms ? r : -1; }
};
template <>
struct FoldRow<float2> {
  static constexpr int stride(int m, int p, int) { return m2l_dd_off(m, p + 1); }
  __host__ __device__ static constexpr int coef(int m, int, int, int r) {
    int o = m, k = 0;
    while (r >= 2 * o + 2) r -= 2 * o + 2, k += 2 * o + 1, ++o;
    return r < 2 * o + 1 ? k + r : -1;
  }
};
// What the translation relies on: coefficient k of order o at m2l_dd_off(m, o) + k,
// an even position each, and nothing else in the row.
constexpr bool m2l_dd_rows_hold(int m, int p) {
  int used = 0;
  for (int o = m; o <= p; ++o) {
    const int n = nred(o) - nred(o - 1), at = m2l_dd_off(m, o);
    if (at & 1) return false;
    for (int k = 0; k < n; ++k, ++used)
      if (FoldRow<float2>::coef(m, p, 0, at + k) != nred(o - 1) - nred(m - 1) + k) return false;
  }
  for (int r = 0; r < m2l_dd_off(m, p + 1); ++r) used -= FoldRow<float2>::coef(m, p, 0, r) >= 0;
  return used == 0;
}
// Folded rows of the cells, FOLD_LANES threads a cell.  A cell with upward tasks
// is the sum of its task partials in order: added up here, not in a launch of its
// own (one of seven in the far-field chain, which is the longer path of small
// systems: a mixed solve of 4,200 sites 1.5 % faster).
constexpr int FOLD_CELLS = 4, FOLD_LANES = 64;
constexpr int nfull(int m, int p) {  // multipoles of orders m..p
  return (p + 1) * (p + 2) * (p + 3) / 6 - m * (m + 1) * (m + 2) / 6;
}
#define CPPE_DEF_FOLD(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                                 \
  template <typename T, typename O>                                                          \
  __global__ void __launch_bounds__(FOLD_CELLS * FOLD_LANES)                                 \
  k_m2l_fold_##NAME(int ncells, const T* __restrict__ M, int mstride,                        \
                                    O* __restrict__ Mr,                                      \
                                    const int* __restrict__ cell_seg,                        \
                                    const int* __restrict__ seg_done,                        \
                    const int* __restrict__ task_ptr, const T* __restrict__ Mpart) {         \
    constexpr int RS = FoldRow<O>::stride(MM, PP, MS);                                       \
    __shared__ T s_m[FOLD_CELLS][nfull(MM, PP)];                                             \
    const int g = threadIdx.x / FOLD_LANES, r0 = threadIdx.x % FOLD_LANES;                   \
    const int cell  = blockIdx.x * FOLD_CELLS + g;                                           \
    /* (a batch's masked segment: its rows are not read) */                                  \
    const bool live = cell < ncells && !(seg_done && seg_done[cell_seg[cell]]);              \
    if (live) {                                                                              \
      const int t0 = task_ptr ? task_ptr[cell] : 0, t1 = task_ptr ? task_ptr[cell + 1] : 0;  \
      for (int r = r0; r < nfull(MM, PP); r += FOLD_LANES) {                                 \
        T v = T(0);                                                                          \
        if (t0 == t1) v = M[(size_t)cell * mstride + r];                                     \
        for (int t = t0; t < t1; ++t) v += Mpart[(size_t)t * mstride + r];                   \
        s_m[g][r] = v;                                                                       \
      }                                                                                      \
    }                                                                                        \
    __syncthreads();                                                                         \
    if (!live) return;                                                                       \
    for (int pos = r0; pos < RS; pos += FOLD_LANES) {                                        \
      T v = T(0);                                                                            \
      const int row = FoldRow<O>::coef(MM, PP, MS, pos);                                     \
      if (row >= 0) {                                                                        \
        _Pragma("unroll") for (int i = 0; i < (FW); ++i) {                                   \
          const int f = m2l_fold_##NAME[row][i][1];                                          \
          if (f != 0) v = fma(T(f), s_m[g][m2l_fold_##NAME[row][i][0]], v);                  \
        }                                                                                    \
      }                                                                                      \
      m2l_store(Mr[(size_t)cell * RS + pos], v);                                             \
    }                                                                                        \
  }
CPPE_M2L_REDUCED(CPPE_DEF_FOLD)
#undef CPPE_DEF_FOLD

// Sums of N per-lane values over the warp, scattered: every step halves the
// values a lane still holds (the lanes with the bit set keep the second half), so
// 36 values take 37 exchanges instead of 180.  Afterwards v[0..cnt) of a lane are
// the sums of values base, base + 1, ...; the order of the additions is fixed.
__device__ __forceinline__ float m2l_xor(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double m2l_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ dd m2l_xor(dd v, int o) { return {m2l_xor(v.h, o), m2l_xor(v.l, o)}; }
__device__ __forceinline__ float m2l_add(float a, float b) { return a + b; }
__device__ __forceinline__ double m2l_add(double a, double b) { return a + b; }
__device__ __forceinline__ dd m2l_add(dd a, dd b) { return dd_add(a, b); }
template <int N, int OFF, typename V>
__device__ __forceinline__ void m2l_scatter(V* v, int lane, int& base, int& cnt) {
  constexpr int h = (N + 1) / 2;
  const bool up   = lane & OFF;
#pragma unroll
  for (int i = 0; i < h; ++i) {
    V keep = v[i], send = v[i];
    if (h + i < N) {
      keep = up ? v[h + i] : v[i];
      send = up ? v[i] : v[h + i];
    }
    // (an unpaired value goes to the lower lanes only)
    const V got = m2l_xor(send, OFF);
    v[i]        = m2l_add(keep, got);
  }
  base += up ? h : 0;
  cnt = up ? max(cnt - h, 0) : min(cnt, h);
  if constexpr (OFF > 1) m2l_scatter<h, OFF / 2>(v, lane, base, cnt);
}

// Asynchronous copy of 8 bytes to shared memory.
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src));
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// (The FP32 kernel's source rows read directly: copied to shared memory by the
// whole warp with cp.async, the L1 wavefronts fell by two thirds and the time
// rose from 0.61 to 0.71 ms at 300,000 sites, the copies' instructions costing
// more than the scattered loads.)
#define CPPE_DEF_M2L_KERNEL(M, P, NAME, NT, LS, MS, FW, UW, FLS)                           \
  template <typename T, bool PRE>                                                          \
  __global__ void __launch_bounds__(128, sizeof(T) == 4 ? 4 : ((P) == 5 ? 2 : 1))          \
        k_m2l_##NAME(TreeView tv, const int4* __restrict__ chunks, int nchunks,            \
                     const T* __restrict__ Mr, T* __restrict__ Lpart,                      \
                     const int* __restrict__ cell_seg, const int* __restrict__ seg_done,   \
                     const T* __restrict__ Dtab, const int* __restrict__ vid) {            \
    const int lane = threadIdx.x & 31;                                                     \
    const int w    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;                         \
    if (w >= nchunks) return;                                                              \
    const int4 ch = chunks[w];                                                             \
    const int A   = ch.x;                                                                  \
    if (seg_done && seg_done[cell_seg[A]]) return; /* finished segment of a batch */       \
    T acc[LS];                                                                             \
    _Pragma("unroll") for (int q = 0; q < LS; ++q) acc[q] = T(0);                          \
    const double4_32a cA = tv.center[A];                                                   \
    for (int idx = ch.y + lane; idx < ch.z; idx += 32) {                                   \
      const int B = tv.m2l_src[idx];                                                       \
      const T* Mb = static_cast<const T*>(                                                 \
            __builtin_assume_aligned(Mr + (size_t)B * m_stride(MS), 16));                  \
      if constexpr (PRE) {                                                                 \
        const T* Dv = static_cast<const T*>(                                               \
              __builtin_assume_aligned(Dtab + (size_t)vid[idx] * (NT), 16));               \
        m2l_##NAME##_pre<T>(Dv, Mb, acc);                                                  \
      } else {                                                                             \
        const double4_32a cB = tv.center[B];                                               \
        m2l_##NAME<T>((T)(cA.x - cB.x), (T)(cA.y - cB.y), (T)(cA.z - cB.z), Mb, acc);      \
      }                                                                                    \
    }                                                                                      \
    int first = 0, cnt = LS;                                                               \
    m2l_scatter<LS, 16>(acc, lane, first, cnt);                                            \
    T* LA = Lpart + (size_t)w * (LS) + first;                                              \
    _Pragma("unroll") for (int q = 0; q < (LS + 31) / 32; ++q) if (q < cnt) LA[q] = acc[q]; \
  }

CPPE_M2L_REDUCED(CPPE_DEF_M2L_KERNEL)
#undef CPPE_DEF_M2L_KERNEL

// Double-float variant for the mixed solver's FP64-accurate residual: the
// same chunks, the reduced multipoles as double-float pairs (k_m2l_fold), the
// partial expansions written in FP64.  In double-float the straight-line
// translation is longer than the instruction cache holds, so this kernel runs
// the same contraction in loop form: each lane has the derivative tensor of
// its source in its own slice of shared memory (a row of an odd number of
// pairs: conflict-free), then adds D_{n+k} M_k over the multipole coefficients
// k, order by order, with the local coefficients n unrolled into registers.
// first w-table entry of the multipole coefficients of order ko
constexpr int m2l_wbase(int m, int p, int ko) {
  int b = 0;
  for (int o = m; o < ko; ++o) b += (nred(o) - nred(o - 1)) * nred(p - o);
  return b;
}
#define CPPE_CHECK_ROWS(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                               \
  static_assert((NT) % 2 == 0, "FP64 tensors are read in 16-byte loads");                   \
  static_assert(m2l_dd_rows_hold(MM, PP), "double-float rows");                             \
  static_assert(m2l_wbase(MM, PP, (PP) + 1) == sizeof(m2l_w_##NAME), "one entry per term"); \
  static_assert((LS) == nred((PP) - (MM)) && (MS) == nred(PP) - nred((MM) - 1), "reduced rows");
CPPE_M2L_REDUCED(CPPE_CHECK_ROWS)
#undef CPPE_CHECK_ROWS

// The multipole coefficients of order KO of a lane's source, all loads in
// flight at once.
template <int M, int KO>
__device__ __forceinline__ void m2l_load_dd(const float2* __restrict__ Mb, float2* mv) {
  const float4* q = reinterpret_cast<const float4*>(Mb + m2l_dd_off(M, KO));
#pragma unroll
  for (int i = 0; i < KO + 1; ++i) {
    const float4 t = q[i];
    mv[2 * i] = make_float2(t.x, t.y), mv[2 * i + 1] = make_float2(t.z, t.w);
  }
}
// mv: the coefficients of order KO, loaded while the previous order was
// contracted (one exposed load latency per translation instead of one per
// coefficient).  A loop over k that picks mv[k] by selects: unrolled code is
// longer than the instruction cache holds.
template <int M, int P, int KO, typename WT>
__device__ __forceinline__ void m2l_contract_dd(const float2* __restrict__ D,
                                                const float2* __restrict__ Mb,
                                                const float2* mv, WT wtab, dd* acc) {
  constexpr int R = nred(P - KO), K = nred(KO) - nred(KO - 1);
  constexpr int base = m2l_wbase(M, P, KO);
  float2 nx[KO < P ? 2 * KO + 4 : 1];
  if constexpr (KO < P) m2l_load_dd<M, KO + 1>(Mb, nx);
  if constexpr (R == 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float2 d = D[wtab(base + k)];
      acc[0]         = dd_fma_lazy(dd{d.x, d.y}, dd{mv[k].x, mv[k].y}, acc[0]);
    }
  } else {
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
      float2 m = mv[0];
#pragma unroll
      for (int i = 1; i < K; ++i) m = k == i ? mv[i] : m;
#pragma unroll
      for (int n = 0; n < R; ++n) {
        const float2 d = D[wtab(base + k * R + n)];
        acc[n]         = dd_fma_lazy(dd{d.x, d.y}, dd{m.x, m.y}, acc[n]);
      }
    }
  }
  if constexpr (KO < P) m2l_contract_dd<M, P, KO + 1>(D, Mb, nx, wtab, acc);
}

// TAB: tensors read from the table; else (vectors off the grid) built per entry.
#define CPPE_DEF_M2L_DD_KERNEL(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                       \
  template <bool TAB>                                                                       \
  __global__ void __launch_bounds__(64, TAB ? ((PP) == 5 ? 8 : 6) : 1)                      \
        k_m2l_##NAME##_dd(TreeView tv, const int4* __restrict__ chunks, int nchunks,        \
                          const float2* __restrict__ Mdd, double* __restrict__ Lpart,       \
                          const float2* __restrict__ Dtab, const int* __restrict__ vid) {   \
    constexpr int DS = (NT) | 1;                                                            \
    __shared__ float2 s_D[2 * 32 * DS];                                                     \
    const int lane = threadIdx.x & 31;                                                      \
    const int w    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;                          \
    if (w >= nchunks) return;                                                               \
    float2* D     = s_D + (threadIdx.x >> 5) * 32 * DS + lane * DS;                         \
    const int4 ch = chunks[w];                                                              \
    dd acc[LS];                                                                             \
    _Pragma("unroll") for (int q = 0; q < LS; ++q) acc[q] = dd{0.f, 0.f};                   \
    const double4_32a cA = tv.center[ch.x];                                                 \
    auto wtab = [](int i) { return (int)m2l_w_##NAME[i]; };                                 \
    for (int base = ch.y; base < ch.z; base += 32) {                                        \
      const int cnt = min(32, ch.z - base), idx = base + min(lane, cnt - 1);                \
      const int B   = tv.m2l_src[idx];                                                      \
      const float2* Mb = static_cast<const float2*>(__builtin_assume_aligned(               \
            Mdd + (size_t)B * FoldRow<float2>::stride(MM, PP, MS), 16));                    \
      float2 mv[2 * (MM) + 2];                                                              \
      m2l_load_dd<MM, MM>(Mb, mv);                                                          \
      if constexpr (TAB) {                                                                  \
        /* the tabulated tensors of the round's vectors, row by row by the whole warp */    \
        const int v = vid[idx];                                                             \
        __syncwarp();                                                                       \
        _Pragma("unroll 4") for (int r = 0; r < cnt; ++r) {                                 \
          const float2* Dv = Dtab + (size_t)__shfl_sync(0xffffffffu, v, r) * (NT);          \
          float2* o        = D - (lane - r) * DS;                                           \
          _Pragma("unroll") for (int i = 0; i < (NT); i += 32) if (i + lane < (NT))         \
                cp_async8(o + i + lane, Dv + i + lane);                                     \
        }                                                                                   \
        cp_async_wait();                                                                    \
        __syncwarp();                                                                       \
      } else {                                                                              \
        /* off the grid of tabulated vectors: the tensor built here */                      \
        const double4_32a cB = tv.center[B];                                                \
        ddv t[NT];                                                                          \
        dtensor_##NAME<ddv>(ddv(dd_from(cA.x - cB.x)), ddv(dd_from(cA.y - cB.y)),           \
                            ddv(dd_from(cA.z - cB.z)), t);                                  \
        _Pragma("unroll") for (int j = 0; j < (NT); ++j) D[j] = make_float2(t[j].h, t[j].l); \
      }                                                                                     \
      if (lane < cnt) m2l_contract_dd<MM, PP, MM>(D, Mb, mv, wtab, acc);                    \
    }                                                                                       \
    int first = 0, cnt = LS;                                                                \
    m2l_scatter<LS, 16>(acc, lane, first, cnt);                                             \
    double* LA = Lpart + (size_t)w * (LS) + first;                                          \
    _Pragma("unroll") for (int q = 0; q < (LS + 31) / 32; ++q) if (q < cnt)                 \
          LA[q] = dd_to(acc[q]);                                                            \
  }

CPPE_M2L_REDUCED(CPPE_DEF_M2L_DD_KERNEL)
#undef CPPE_DEF_M2L_DD_KERNEL

// The full local expansion of every cell (FLS rows) from the reduced partial
// expansions of its chunks (LS rows), summed in order; 0 without chunks.
#define CPPE_DEF_LSUM(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                                  \
  template <typename T>                                                                       \
  __global__ void k_lsum_##NAME(int ncells, const int* __restrict__ cell_chunk_ptr,           \
                                const T* __restrict__ Lpart, T* __restrict__ L,               \
                                const int* __restrict__ cell_seg,                             \
                                const int* __restrict__ seg_done) {                           \
    const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;                             \
    const int cell = (int)(gid / (FLS)), row = (int)(gid % (FLS));                            \
    if (cell >= ncells) return;                                                               \
    if (seg_done && seg_done[cell_seg[cell]]) return; /* a batch's masked segment */          \
    const int t0 = cell_chunk_ptr[cell], t1 = cell_chunk_ptr[cell + 1];                       \
    T v = T(0);                                                                               \
    _Pragma("unroll") for (int i = 0; i < (UW); ++i) {                                        \
      const int f = m2l_unfold_##NAME[row][i][1];                                             \
      if (f == 0) continue;                                                                   \
      const T* q = Lpart + m2l_unfold_##NAME[row][i][0];                                      \
      T acc = T(0);                                                                           \
      for (int t = t0; t < t1; ++t) acc += q[(size_t)t * (LS)];                               \
      v = fma(T(f), acc, v);                                                                  \
    }                                                                                         \
    L[(size_t)cell * (FLS) + row] = v;                                                        \
  }
CPPE_M2L_REDUCED(CPPE_DEF_LSUM)
#undef CPPE_DEF_LSUM

// Runs the fixed-order translation when one is compiled for (m, p): fold, a
// warp per chunk of at most M2L_CHUNK sources of one target cell (so that the
// GPU holds several warps per cell), the per-cell sums.  DD: in double-float
// (Mr as float2).  Returns false otherwise.
template <bool DD, typename T, typename O>
bool launch_m2l_fixed(const TreeView& tv, int m, int p, const int4* chunks, int nchunks,
                      const int* cell_chunk_ptr, const T* M, int mstride, DBuf<O>& Mr,
                      DBuf<T>& Lpart, T* L, cudaStream_t s, const int* cell_seg, const int* seg_done,
                      const void* dtab, const int* vid, const int* task_ptr,
                      const T* Mpart) {
  bool ok = false;
  auto grid = [](long work, int b) { return (unsigned)((work + b - 1) / b); };
#define CPPE_LAUNCH_M2L(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                                 \
  if constexpr ((MM) == 1 || (!DD && sizeof(T) == 8))                                          \
  if (!ok && m == MM && p == PP) {                                                             \
    ok = true;                                                                                 \
    constexpr int RS = FoldRow<O>::stride(MM, PP, MS);                                         \
    Mr.alloc((size_t)std::max(1, tv.ncells) * RS);                                             \
    Lpart.alloc((size_t)std::max(1, nchunks) * (LS));                                          \
    if (nchunks > 0) {                                                                         \
      k_m2l_fold_##NAME<T, O><<<grid(tv.ncells, FOLD_CELLS), FOLD_CELLS * FOLD_LANES, 0, s>>>(  \
            tv.ncells, M, mstride, Mr.p, cell_seg, seg_done, task_ptr, Mpart);                 \
      CG_LAUNCH();                                                                             \
      if constexpr (DD) {                                                                      \
        const unsigned b = grid((long)nchunks * 32, 64);                                       \
        const float2* dt = (const float2*)dtab;                                                \
        if (dt)                                                                                \
          k_m2l_##NAME##_dd<true><<<b, 64, 0, s>>>(tv, chunks, nchunks, Mr.p, Lpart.p, dt,     \
                                                   vid);                                       \
        else                                                                                   \
          k_m2l_##NAME##_dd<false><<<b, 64, 0, s>>>(tv, chunks, nchunks, Mr.p, Lpart.p,        \
                                                    nullptr, nullptr);                         \
      } else if (sizeof(T) == 8 && dtab) {                                                     \
        if constexpr (sizeof(T) == 8)                                                          \
          k_m2l_##NAME<T, true><<<grid((long)nchunks * 32, 128), 128, 0, s>>>(                 \
                tv, chunks, nchunks, Mr.p, Lpart.p, cell_seg, seg_done, (const T*)dtab, vid);  \
      } else {                                                                                 \
        k_m2l_##NAME<T, false><<<grid((long)nchunks * 32, 128), 128, 0, s>>>(                  \
              tv, chunks, nchunks, Mr.p, Lpart.p, cell_seg, seg_done, nullptr, nullptr);       \
      }                                                                                        \
      CG_LAUNCH();                                                                             \
    }                                                                                          \
    if (tv.ncells > 0) {                                                                       \
      k_lsum_##NAME<T><<<grid((long)tv.ncells * (FLS), 256), 256, 0, s>>>(                     \
            tv.ncells, cell_chunk_ptr, Lpart.p, L, cell_seg, seg_done);                        \
      CG_LAUNCH();                                                                             \
    }                                                                                          \
  }
  CPPE_M2L_REDUCED(CPPE_LAUNCH_M2L)
#undef CPPE_LAUNCH_M2L
  return ok;
}

}  // namespace cg
