// M2L with the expansion order fixed at compile time (the orders the
// benchmark configurations use; other orders take the table-driven k_m2l).
//
// Same operator as k_m2l (src/core/fmm/calculate.cc:186-203 with the
// field_m*.cc M2L kernels), organised for registers: each lane of a warp
// takes its own source cell of the target's interaction list, evaluates the
// straight-line translation generated by gen_m2l.py (derivative tensor and
// partial local expansion in registers, the source multipole streamed one
// coefficient at a time), and the lanes' partial expansions are added with
// warp shuffles in a fixed order at the end.
//
// The translation works between harmonic-reduced coefficients (z-power 0 or 1,
// see gen_m2l.py): k_m2l_fold turns each cell's multipole into its reduced row
// before, k_lsum gives back the full local expansion after.  Measured (M2L
// phase with folding and per-cell sums, 300,000 sites order 6, 14.6 M
// translations, full coefficients against reduced): MEASURED_M2L
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
#define CPPE_DEF_DTAB(MM, PP, NAME, NT, LS, MS, FW, UW, FLS, FMS)                           \
  template <typename T>                                                                     \
  __global__ void k_dtab_##NAME(int nvec, const double4_32a* __restrict__ vec,              \
                                T* __restrict__ D) {                                        \
    const int v = blockIdx.x * blockDim.x + threadIdx.x;                                    \
    if (v >= nvec) return;                                                                  \
    const double4_32a r = vec[v];                                                           \
    dtensor_##NAME<T>((T)r.x, (T)r.y, (T)r.z, D + (size_t)v * (NT));                        \
  }                                                                                         \
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
template <typename T>
const void* m2l_dtab(const Geometry& g, int m, int p, FieldWork<T>& w, bool dd, cudaStream_t s) {
  const int nv = (int)g.h_vec.size();
  if (nv == 0) return nullptr;
  const void* out = nullptr;
#define CPPE_BUILD_DTAB(MM, PP, NAME, NT, LS, MS, FW, UW, FLS, FMS)                          \
  if (!out && m == MM && p == PP) {                                                          \
    const size_t cnt = (size_t)nv * (NT);                                                    \
    if (dd) {                                                                                \
      if (w.dtab_dd.n != cnt) {                                                              \
        w.dtab_dd.alloc(cnt);                                                                \
        k_dtab_##NAME##_dd<<<(nv + 63) / 64, 64, 0, s>>>(nv, g.vec.p, w.dtab_dd.p);          \
        CG_LAUNCH();                                                                         \
      }                                                                                      \
      out = w.dtab_dd.p;                                                                     \
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
// ones (stride m_stride(FMS)); thread per (cell, reduced row).  To double-float
// pairs for the double-float translation (sums in T).
__device__ __forceinline__ void m2l_store(float& o, float v) { o = v; }
__device__ __forceinline__ void m2l_store(double& o, double v) { o = v; }
__device__ __forceinline__ void m2l_store(float2& o, double v) {
  const float h = (float)v;
  o             = make_float2(h, (float)(v - (double)h));
}
#define CPPE_DEF_FOLD(MM, PP, NAME, NT, LS, MS, FW, UW, FLS, FMS)                            \
  template <typename T, typename O>                                                          \
  __global__ void k_m2l_fold_##NAME(int ncells, const T* __restrict__ M, O* __restrict__ Mr, \
                                    const int* __restrict__ cell_seg,                        \
                                    const int* __restrict__ seg_done) {                      \
    constexpr int RS = m_stride(MS);                                                         \
    const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;                            \
    const int cell = (int)(gid / RS), row = (int)(gid % RS);                                 \
    if (cell >= ncells) return;                                                              \
    if (seg_done && seg_done[cell_seg[cell]]) return; /* a batch's masked segment */         \
    T v = T(0);                                                                              \
    if (row < (MS)) {                                                                        \
      const T* m = M + (size_t)cell * m_stride(FMS);                                         \
      _Pragma("unroll") for (int i = 0; i < (FW); ++i) {                                     \
        const int f = m2l_fold_##NAME[row][i][1];                                            \
        if (f != 0) v = fma(T(f), m[m2l_fold_##NAME[row][i][0]], v);                         \
      }                                                                                      \
    }                                                                                        \
    m2l_store(Mr[(size_t)cell * RS + row], v);                                               \
  }
CPPE_M2L_REDUCED(CPPE_DEF_FOLD)
#undef CPPE_DEF_FOLD

#define CPPE_DEF_M2L_KERNEL(M, P, NAME, NT, LS, MS, FW, UW, FLS, FMS)                      \
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
    _Pragma("unroll") for (int q = 0; q < LS; ++q) {                                       \
      T v = acc[q];                                                                        \
      _Pragma("unroll") for (int off = 16; off > 0; off >>= 1) v +=                        \
            __shfl_xor_sync(0xffffffffu, v, off);                                          \
      acc[q] = v;                                                                          \
    }                                                                                      \
    T* LA = Lpart + (size_t)w * (LS);                                                      \
    _Pragma("unroll") for (int q = 0; q < LS; ++q) if ((q & 31) == lane) LA[q] = acc[q];   \
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
template <int M, int P, int KO, typename WT>
__device__ __forceinline__ void m2l_contract_dd(const float2* __restrict__ D,
                                                const float2* __restrict__ Mb, WT wtab,
                                                dd* acc) {
  constexpr int R = nred(P - KO), k0 = nred(KO - 1), k1 = nred(KO);
  constexpr int base = m2l_wbase(M, P, KO), moff = nred(M - 1);
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const float2 mv = Mb[k - moff];
    const int wr    = base + (k - k0) * R;
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const float2 d = D[wtab(wr + n)];
      acc[n]         = dd_fma_lazy(dd{d.x, d.y}, dd{mv.x, mv.y}, acc[n]);
    }
  }
  if constexpr (KO < P) m2l_contract_dd<M, P, KO + 1>(D, Mb, wtab, acc);
}

// TAB: tensors read from the table; else (vectors off the grid) built per entry.
#define CPPE_DEF_M2L_DD_KERNEL(MM, PP, NAME, NT, LS, MS, FW, UW, FLS, FMS)                  \
  template <bool TAB>                                                                       \
  __global__ void __launch_bounds__(64)                                                     \
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
    for (int idx = ch.y + lane; idx < ch.z; idx += 32) {                                    \
      const int B = tv.m2l_src[idx];                                                        \
      const float2* Mb = static_cast<const float2*>(                                        \
            __builtin_assume_aligned(Mdd + (size_t)B * m_stride(MS), 16));                  \
      if constexpr (TAB) {                                                                  \
        /* the tabulated tensor of this entry's vector into the lane's row */               \
        const float4* Dv = reinterpret_cast<const float4*>(Dtab + (size_t)vid[idx] * (NT)); \
        _Pragma("unroll 8") for (int i = 0; i < (NT) / 2; ++i) {                            \
          const float4 t = Dv[i];                                                           \
          D[2 * i]       = make_float2(t.x, t.y);                                           \
          D[2 * i + 1]   = make_float2(t.z, t.w);                                           \
        }                                                                                   \
      } else {                                                                              \
        /* off the grid of tabulated vectors: the tensor built here */                      \
        const double4_32a cB = tv.center[B];                                                \
        ddv t[NT];                                                                          \
        dtensor_##NAME<ddv>(ddv(dd_from(cA.x - cB.x)), ddv(dd_from(cA.y - cB.y)),           \
                            ddv(dd_from(cA.z - cB.z)), t);                                  \
        _Pragma("unroll") for (int j = 0; j < (NT); ++j) D[j] = make_float2(t[j].h, t[j].l); \
      }                                                                                     \
      m2l_contract_dd<MM, PP, MM>(D, Mb, wtab, acc);                                        \
    }                                                                                       \
    double* LA = Lpart + (size_t)w * (LS);                                                  \
    _Pragma("unroll") for (int q = 0; q < LS; ++q) {                                        \
      dd v = acc[q];                                                                        \
      _Pragma("unroll") for (int off = 16; off > 0; off >>= 1) {                            \
        const dd o{__shfl_xor_sync(0xffffffffu, v.h, off),                                  \
                   __shfl_xor_sync(0xffffffffu, v.l, off)};                                 \
        v = dd_add(v, o);                                                                   \
      }                                                                                     \
      if ((q & 31) == lane) LA[q] = dd_to(v);                                               \
    }                                                                                       \
  }

CPPE_M2L_REDUCED(CPPE_DEF_M2L_DD_KERNEL)
#undef CPPE_DEF_M2L_DD_KERNEL

// The full local expansion of every cell (FLS rows) from the reduced partial
// expansions of its chunks (LS rows), summed in order; 0 without chunks.
#define CPPE_DEF_LSUM(MM, PP, NAME, NT, LS, MS, FW, UW, FLS, FMS)                             \
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
                      const int* cell_chunk_ptr, const T* M, DBuf<O>& Mr, DBuf<T>& Lpart, T* L,
                      cudaStream_t s, const int* cell_seg, const int* seg_done,
                      const void* dtab, const int* vid) {
  bool ok = false;
  auto grid = [](long work, int b) { return (unsigned)((work + b - 1) / b); };
#define CPPE_LAUNCH_M2L(MM, PP, NAME, NT, LS, MS, FW, UW, FLS, FMS)                            \
  if (!ok && m == MM && p == PP) {                                                             \
    ok = true;                                                                                 \
    Mr.alloc((size_t)std::max(1, tv.ncells) * m_stride(MS));                                   \
    Lpart.alloc((size_t)std::max(1, nchunks) * (LS));                                          \
    if (nchunks > 0) {                                                                         \
      k_m2l_fold_##NAME<T, O><<<grid((long)tv.ncells * m_stride(MS), 256), 256, 0, s>>>(       \
            tv.ncells, M, Mr.p, cell_seg, seg_done);                                           \
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
