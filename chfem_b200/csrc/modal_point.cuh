// modal_point.cuh -- the pointwise PCG pass of models whose operator passes run in voxel modes
// (stencil_modal.cuh) and of 2D models, for one right-hand side or a block of NR: r -= alpha q, delta = r . M^-1 r,
// the stopping test, and x += alpha d.
//
// The solution is updated every second iteration.  d alternates between two buffers, so after an
// odd pass both of the pair's directions are still there: the even pass (XM = 0) leaves x alone
// and records its step in the scalar record (xa), the odd one (XM = 1) adds both,
// x += xa d_old + alpha d, in the order and with the rounding of two updates.  A right-hand side
// that stops in an even pass gets its pending step from the odd pass that follows it in the same
// graph.  FP64 x is 16 of the 48 bytes per unknown (FP64; 16 of 32 with FP32 fields) that a pass
// with x moves; deferred, two passes move 24 + 56 bytes instead of 96 (12 + 36 instead of 64).
// XM = 2: x updated in every pass, with the max-norms (the infinity and error norms read them).
//
// Each thread moves 16 bytes of every vector at a time (VW words; a block whose vectors do not all
// start on 16 bytes takes the widest words that they all start on).  The Jacobi diagonal comes from the table by material
// counts instead of 8 element-matrix diagonals and a division per node.
#pragma once
#include "stencil_modal.cuh"
#include "pointwise.cuh"

namespace chfem {

template <typename T>
struct MdPw {
  double* x; const T* d; const T* dold; T* r; const T* q;  // [NR][n]
  const uint16_t* keys;
  const T* tab;        // the table of the voxel modes: inverse diagonal by material counts
  const double* invd;  // scalar density field, 2D models: the inverse diagonal per unknown (keys, tab unused)
  int nmat;
  long n;
  DevScalars* sc;      // [NR]
  RedCtl rc;
  SolveCfg cfg;
};

constexpr int MP_NT = 256;

template <typename T, int VW>
__device__ __forceinline__ void mp_ld(const T* p, T (&v)[VW]) {
  if constexpr (VW == 4) { const float4 t = *reinterpret_cast<const float4*>(p); v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
  else if constexpr (VW == 2 && sizeof(T) == 8) { const double2 t = *reinterpret_cast<const double2*>(p); v[0] = t.x; v[1] = t.y; }
  else if constexpr (VW == 2) { const float2 t = *reinterpret_cast<const float2*>(p); v[0] = t.x; v[1] = t.y; }
  else v[0] = *p;
}
template <typename T, int VW>
__device__ __forceinline__ void mp_st(T* p, const T (&v)[VW]) {
  if constexpr (VW == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if constexpr (VW == 2 && sizeof(T) == 8) *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  else if constexpr (VW == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else *p = v[0];
}
// FP64 x of VW unknowns, read and written once per pair of iterations (no reuse: streamed)
template <int VW>
__device__ __forceinline__ void mp_ldx(const double* p, double (&v)[VW]) {
  if constexpr (VW == 1) v[0] = __ldcs(p);
  else
#pragma unroll
    for (int i = 0; i < VW; i += 2) { const double2 t = __ldcs(reinterpret_cast<const double2*>(p + i)); v[i] = t.x; v[i + 1] = t.y; }
}
template <int VW>
__device__ __forceinline__ void mp_stx(double* p, const double (&v)[VW]) {
  if constexpr (VW == 1) __stcs(p, v[0]);
  else
#pragma unroll
    for (int i = 0; i < VW; i += 2) __stcs(reinterpret_cast<double2*>(p + i), make_double2(v[i], v[i + 1]));
}

template <int ND, typename T, int NR, int XM, int VW>
__global__ void __launch_bounds__(MP_NT) k_md_point(MdPw<T> a) {
  constexpr int NV = XM == 2 ? 4 : 1;  // reduced values per right-hand side
  __shared__ double sred[MP_NT / 32];
  __shared__ T sTab[MD_NCOUNT];
  bool done[NR];
  double alpha[NR], xa[NR];
  bool all = true;
#pragma unroll
  for (int k = 0; k < NR; k++) {
    const double al = a.sc[k].alpha;  // read beside done, not after it
    done[k] = a.sc[k].done;
    xa[k] = XM == 1 ? a.sc[k].xa : 0.0;
    alpha[k] = done[k] ? 0.0 : al;
    all = all && done[k] && xa[k] == 0.0;
  }
  const int tid = threadIdx.x;
  const bool pre = a.cfg.precond != 0, two = a.nmat <= 2;
  if (pre && !a.invd)
    for (int i = tid; i < (two ? 9 : MD_NCOUNT); i += MP_NT) sTab[i] = a.tab[i];
  if (all) return;
  __syncthreads();
  double vals[NV * NR];
#pragma unroll
  for (int k = 0; k < NV * NR; k++) vals[k] = 0.0;
  // unknowns j0 .. j0 + W - 1 of every right-hand side
  auto chunk = [&](long j0, auto width) {
    constexpr int W = decltype(width)::value;
    T inv[W];
    if (!pre) {
#pragma unroll
      for (int i = 0; i < W; i++) inv[i] = T(1);
    } else if (a.invd) {
#pragma unroll
      for (int i = 0; i < W; i++) inv[i] = T(a.invd[j0 + i]);
    } else if constexpr (ND == 1) {
#pragma unroll
      for (int i = 0; i < W; i++) inv[i] = sTab[md_count_index(a.keys[j0 + i], two)];
    } else {  // the unknowns span at most two nodes
      const long node = j0 / ND;
      const int c = (int)(j0 - node * ND);
      const T i0 = sTab[md_count_index(a.keys[node], two)];
      T i1 = i0;
      if (W > 1 && c + W > ND) i1 = sTab[md_count_index(a.keys[node + 1], two)];
#pragma unroll
      for (int i = 0; i < W; i++) inv[i] = c + i < ND ? i0 : i1;
    }
#pragma unroll
    for (int k = 0; k < NR; k++) {
      const long j = k * a.n + j0;
      if (NR > 1 && done[k] && (XM != 1 || xa[k] == 0.0)) continue;
      if constexpr (XM != 0) {
        T dv[W];
        [[maybe_unused]] T dp[W];
        double xv[W];
        mp_ldx<W>(a.x + j, xv);
        if constexpr (XM == 1) {
          mp_ld<T, W>(a.dold + j, dp);
#pragma unroll
          for (int i = 0; i < W; i++) xv[i] = fma(xa[k], (double)dp[i], xv[i]);
        }
        if (XM == 2 || !done[k]) {
          mp_ld<T, W>(a.d + j, dv);
#pragma unroll
          for (int i = 0; i < W; i++) xv[i] = fma(alpha[k], (double)dv[i], xv[i]);
        }
        mp_stx<W>(a.x + j, xv);
        if constexpr (XM == 2) {
#pragma unroll
          for (int i = 0; i < W; i++) {
            vals[NV * k + 2] = fmax(vals[NV * k + 2], fabs((double)dv[i]));
            vals[NV * k + 3] = fmax(vals[NV * k + 3], fabs(xv[i]));
          }
        }
      }
      if (done[k]) continue;
      const T al = T(alpha[k]);
      T rv[W], qv[W];
      mp_ld<T, W>(a.r + j, rv);
      mp_ld<T, W>(a.q + j, qv);
#pragma unroll
      for (int i = 0; i < W; i++) {
        rv[i] = fma(-al, qv[i], rv[i]);
        vals[NV * k] += (double)rv[i] * (double)(rv[i] * inv[i]);
        if constexpr (XM == 2) vals[NV * k + 1] = fmax(vals[NV * k + 1], fabs((double)rv[i]));
      }
      mp_st<T, W>(a.r + j, rv);
    }
  };
  const long nv = a.n / VW;
  for (long t = blockIdx.x * (long)MP_NT + tid; t < nv; t += (long)gridDim.x * MP_NT) chunk(t * VW, std::integral_constant<int, VW>{});
  if constexpr (VW > 1 && NR == 1) {  // the last unknowns, when n is not a multiple of the width
    const long j = nv * VW + tid;
    if (blockIdx.x == 0 && j < a.n) chunk(j, std::integral_constant<int, 1>{});
  }
  bool ismax[NV * NR];
#pragma unroll
  for (int k = 0; k < NV * NR; k++) ismax[k] = (k % NV) != 0;
  double out[NV * NR];
  if (grid_reduce<MP_NT, NV * NR>(vals, ismax, a.rc, blockIdx.x, out, sred) && tid == 0) {
#pragma unroll
    for (int k = 0; k < NR; k++) {
      a.sc[k].xa = (XM == 0 && !done[k]) ? alpha[k] : 0.0;
      if (done[k]) continue;
      double s4[4] = {out[NV * k], 0.0, 0.0, 0.0};
      if constexpr (XM == 2) { s4[1] = out[NV * k + 1]; s4[2] = out[NV * k + 2]; s4[3] = out[NV * k + 3]; }
      for (int t = 0; t < 4; t++) a.sc[k].red[t] = s4[t];
      pcg_finish(PW_PCG, s4, a.sc + k, a.cfg);
    }
  }
}

}  // namespace chfem
