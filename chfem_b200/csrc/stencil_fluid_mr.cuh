// stencil_fluid_mr.cuh -- the passes of (P)MINRES on the Stokes operator (chfem/src/femhmg/
// cudapcg/solvers/pminres.cu:100-204), for one flow direction or the NR directions of a model at
// once (the reference solves them one after the other, femhmg.c:1017-1119).  FP64.
//
// An iteration is three passes:
//   k_fl_mr_dir    d = M^-1 r + beta d, q = s + beta q, and alpha = delta / (q . M^-1 q);
//   k_fl_mr_upd    r -= alpha q, x += alpha d, and z = M^-1 r, stored as one record of 4 doubles
//                  per grid node and direction -- DIM velocities and the pressure; an interface
//                  node's velocities are 0 (no slip), solid nodes' records are never touched;
//                  where the grid is large against its fluid nodes (fl_by_node), per fluid node;
//   k_fl_mr_apply  s = A z, delta = z . s, r . z, the max-norms where the stopping test reads
//                  them, and the finisher (mr_finish).
// The gather over a node's 27 neighbours then loads one 32-byte record each, at constant offsets
// from the node's own (periodic wraps aside): no DOF number on the way, so the loads do not wait
// on one another.  It is bound by their latency.  Measured at 96^3, porosity 0.35, one direction:
// forming z = M^-1 (r - alpha q) in the gather (8 loads of 8 bytes and 4 multiply-adds per
// neighbour) 139 us an iteration, records by DOF number 76 us, by grid node 70 us.  The records of a
// grid cost 32 bytes per node and direction of memory, and no more traffic: a fluid node's
// neighbours within its fluid voxels are fluid nodes.  r is no neighbour input of any pass and is
// updated in place.
//
// The row of a pore node (all its voxels fluid) is summed by neighbour once per model on the
// host: 27 blocks of 4 x 4 (c_flA) instead of 64 (voxel, local node) pairs of them, uniform
// over the warp and so constant-bank operands.  An interface node's pressure row keeps the sum
// over its fluid voxels (matrix_free.cu:926-977).
#pragma once
#include "stencil_fluid.cuh"
#include "minres.cuh"

namespace chfem {

// assembled rows of a pore node: [neighbour][row DIM + 1][column DIM + 1]
__constant__ double c_flA[27 * 16];

struct FlMrArgs {
  double* r; double* q; double* s; double* d; double* x;  // [NR][n]
  double* z;                                              // [nodes or fluid nodes][NR][4]
  const uint32_t* node_of_dof; const uint8_t* bkeys;
  const uint32_t* dof_of_node;  // records per fluid node: their numbers; per grid node: null
  int R, C, L;
  long nV, nB, n;   // n: unknowns per direction
  DevScalars* sc;   // [NR]
  RedCtl rc;
  MrCfg cfg;
  int finish, skip_if_done;
};

// inverse diagonal of unknown j of the vector layout [DIM nV velocities | nV + nB pressures]
template <int DIM>
__device__ __forceinline__ double fl_mr_inv(long j, long nV, const uint8_t* bkeys, const double* sbd, bool pre) {
  if (!pre) return 1.0;
  if (j < DIM * nV) return c_fldiag.pore[j % DIM];
  return j < (DIM + 1) * nV ? c_fldiag.pore[DIM] : sbd[bkeys[j - (DIM + 1) * nV]];
}

// the interface diagonals in shared memory, from an array (constant memory serialises lanes that
// read different entries)
__device__ double d_flborder[256];
__device__ __forceinline__ void fl_mr_table(double* sbd) {
  for (int i = threadIdx.x; i < 256; i += PW_NT) sbd[i] = d_flborder[i];
}

// whether a pass has nothing to do; done[k]: direction k has stopped (its vectors stay)
template <int NR>
__device__ __forceinline__ bool fl_mr_done(const FlMrArgs& a, bool (&done)[NR]) {
  bool all = true;
#pragma unroll
  for (int k = 0; k < NR; k++) { done[k] = a.skip_if_done && a.sc[k].done; all = all && done[k]; }
  return all;
}

template <int NR, int DIM>
__global__ void __launch_bounds__(PW_NT) k_fl_mr_dir(FlMrArgs a) {
  constexpr int U = NR == 1 ? 4 : 2;  // unknowns per thread and step, their loads issued together
  __shared__ double sred[PW_NT / 32];
  __shared__ double sbd[256];
  fl_mr_table(sbd);
  bool done[NR];
  if (fl_mr_done<NR>(a, done)) return;
  double beta[NR], sum[NR];
#pragma unroll
  for (int k = 0; k < NR; k++) { beta[k] = a.sc[k].beta; sum[k] = 0.0; }
  __syncthreads();
  const long step = (long)gridDim.x * PW_NT;
  for (long j0 = blockIdx.x * (long)PW_NT + threadIdx.x; j0 < a.n; j0 += U * step) {
    double inv[U];
#pragma unroll
    for (int u = 0; u < U; u++) inv[u] = j0 + u * step < a.n ? fl_mr_inv<DIM>(j0 + u * step, a.nV, a.bkeys, sbd, a.cfg.precond != 0) : 0.0;
#pragma unroll
    for (int k = 0; k < NR; k++) {
      if (NR > 1 && done[k]) continue;
      double r[U], s[U], d[U], q[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const long i = k * a.n + j0 + u * step;
        const bool in = j0 + u * step < a.n;
        r[u] = in ? a.r[i] : 0.0; s[u] = in ? a.s[i] : 0.0; d[u] = in ? a.d[i] : 0.0; q[u] = in ? a.q[i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const long i = k * a.n + j0 + u * step;
        const double qn = fma(beta[k], q[u], s[u]);
        if (j0 + u * step < a.n) {
          a.d[i] = fma(beta[k], d[u], r[u] * inv[u]);
          a.q[i] = qn;
          sum[k] += qn * (qn * inv[u]);
        }
      }
    }
  }
  const bool ismax[NR] = {};
  double out[NR];
  if (grid_reduce<PW_NT, NR>(sum, ismax, a.rc, blockIdx.x, out, sred) && threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NR; k++)
      if (!done[k]) { a.sc[k].red[5] = out[k]; a.sc[k].alpha = a.sc[k].delta / out[k]; }
  }
}

// finish codes without a step (the initial residual, an initial guess) take alpha = 0
template <int NR, int DIM>
__global__ void __launch_bounds__(PW_NT) k_fl_mr_upd(FlMrArgs a) {
  constexpr int U = NR == 1 ? 4 : 2;
  __shared__ double sbd[256];
  fl_mr_table(sbd);
  bool done[NR];
  if (fl_mr_done<NR>(a, done)) return;
  const bool move = a.finish == FIN_MR_STEP;
  double alpha[NR];
#pragma unroll
  for (int k = 0; k < NR; k++) alpha[k] = move ? a.sc[k].alpha : 0.0;
  __syncthreads();
  const long nVD = DIM * a.nV, step = (long)gridDim.x * PW_NT;
  for (long j0 = blockIdx.x * (long)PW_NT + threadIdx.x; j0 < a.n; j0 += U * step) {
    double inv[U];
    long rec[U];  // the unknown's place in its node's records (direction 0)
    bool edge[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long j = j0 + u * step;
      const bool in = j < a.n, vel = j < nVD;
      const long dof = vel ? j / DIM : j - nVD;
      inv[u] = in ? fl_mr_inv<DIM>(j, a.nV, a.bkeys, sbd, a.cfg.precond != 0) : 0.0;
      rec[u] = in ? (a.dof_of_node ? dof : (long)a.node_of_dof[dof]) * (4 * NR) + (vel ? j - dof * DIM : DIM) : 0;
      edge[u] = !vel && dof >= a.nV;
    }
#pragma unroll
    for (int k = 0; k < NR; k++) {
      if (NR > 1 && done[k]) continue;
      double r[U], q[U], d[U], x[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const long i = k * a.n + j0 + u * step;
        const bool in = j0 + u * step < a.n, m = in && move;
        r[u] = in ? a.r[i] : 0.0; q[u] = m ? a.q[i] : 0.0; d[u] = m ? a.d[i] : 0.0; x[u] = m ? a.x[i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (j0 + u * step >= a.n) continue;
        const long i = k * a.n + j0 + u * step;
        const double rn = fma(-alpha[k], q[u], r[u]);
        if (move) {
          a.r[i] = rn;
          a.x[i] = fma(alpha[k], d[u], x[u]);
        }
        double* z = a.z + rec[u] + 4 * k;
        *z = rn * inv[u];
        if (edge[u]) {  // interface node: no velocity
#pragma unroll
          for (int c = 1; c <= DIM; c++) z[-c] = 0.0;
        }
      }
    }
  }
}

// one 32-byte record (written by an earlier launch)
__device__ __forceinline__ void fl_mr_rec(const double* p, double (&v)[4]) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// voxels e of a node that also hold its neighbour o (pixels: DIM = 2)
template <int DIM>
__host__ __device__ constexpr bool fl_pair(int e, int b, int o) {
  return drow(b) - drow(e) == o % 3 - 1 && dcol(b) - dcol(e) == (o / 3) % 3 - 1 && (DIM == 2 || dlay(b) - dlay(e) == o / 9 - 1);
}
template <int DIM>
__host__ __device__ constexpr unsigned fl_mr_emask(int o) {
  unsigned m = 0;
  for (int e = 0; e < (1 << DIM); e++)
    for (int b = 0; b < (1 << DIM); b++)
      if (fl_pair<DIM>(e, b, o)) m |= 1u << e;
  return m;
}

// MAXN: the stopping test reads max-norms (infinity / error norm).  GRID: records per grid node.
template <int NR, int DIM, bool MAXN, bool GRID>
__global__ void __launch_bounds__(FL_NT, NR == 1 ? 3 : 2) k_fl_mr_apply(FlMrArgs a) {
  constexpr int NE = 1 << DIM, ED = (DIM + 1) * NE, PC = DIM * NE, NO = DIM == 3 ? 27 : 9, D1 = DIM + 1;
  constexpr int NV = MAXN ? 5 : 2;
  __shared__ double sred[FL_NT / 32];
  bool done[NR];
  if (fl_mr_done<NR>(a, done)) return;
  const long nV = a.nV, nT = a.nV + a.nB, n = a.n;
  const unsigned R = (unsigned)a.R, C = (unsigned)a.C, L = (unsigned)a.L, RC = R * C;
  double vals[NV * NR];
#pragma unroll
  for (int k = 0; k < NV * NR; k++) vals[k] = 0.0;
  for (long t = blockIdx.x * (long)FL_NT + threadIdx.x; t < nT; t += (long)gridDim.x * FL_NT) {
    const unsigned node = a.node_of_dof[t];
    const unsigned l = node / RC, cr = node - l * RC, c = cr / R, r = cr - c * R;
    // offsets of the neighbour rows, columns and layers
    const unsigned rr[3] = {r ? r - 1 : R - 1, r, r + 1 < R ? r + 1 : 0};
    const unsigned cc[3] = {(c ? c - 1 : C - 1) * R, c * R, (c + 1 < C ? c + 1 : 0) * R};
    const unsigned ll[3] = {(l ? l - 1 : L - 1) * RC, l * RC, (l + 1 < L ? l + 1 : 0) * RC};
    const bool pore = t < nV;
    double out[NR][D1];
#pragma unroll
    for (int k = 0; k < NR; k++)
#pragma unroll
      for (int i = 0; i < D1; i++) out[k][i] = 0.0;
    if (pore) {
#pragma unroll
      for (int o = 0; o < NO; o++) {
        size_t nb = rr[o % 3] + cc[(o / 3) % 3] + ll[DIM == 3 ? o / 9 : 1];
        if constexpr (!GRID) nb = a.dof_of_node[nb];
#pragma unroll
        for (int k = 0; k < NR; k++) {
          double v[4];
          fl_mr_rec(a.z + (nb * NR + k) * 4, v);
#pragma unroll
          for (int i = 0; i < D1; i++)
#pragma unroll
            for (int m = 0; m < D1; m++) out[k][i] = fma(c_flA[(o * D1 + i) * D1 + m], v[m], out[k][i]);
        }
      }
    } else {
      const unsigned fk = a.bkeys[t - nV];
#pragma unroll
      for (int o = 0; o < NO; o++) {
        if (!(fk & fl_mr_emask<DIM>(o))) continue;
        // coefficients of the pressure row: sum over the node's fluid voxels that hold o
        double g[D1];
#pragma unroll
        for (int m = 0; m < D1; m++) g[m] = 0.0;
#pragma unroll
        for (int e = 0; e < NE; e++)
#pragma unroll
          for (int b = 0; b < NE; b++)
            if (fl_pair<DIM>(e, b, o) && ((fk >> e) & 1u)) {
#pragma unroll
              for (int m = 0; m < DIM; m++) g[m] += c_flK64[(PC + e) * ED + DIM * b + m];
              g[DIM] -= c_flK64[(PC + e) * ED + PC + b];
            }
        size_t nb = rr[o % 3] + cc[(o / 3) % 3] + ll[DIM == 3 ? o / 9 : 1];
        if constexpr (!GRID) nb = a.dof_of_node[nb];
#pragma unroll
        for (int k = 0; k < NR; k++) {
          double v[4];
          fl_mr_rec(a.z + (nb * NR + k) * 4, v);
#pragma unroll
          for (int m = 0; m < D1; m++) out[k][DIM] = fma(g[m], v[m], out[k][DIM]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NR; k++) {
      if (NR > 1 && done[k]) continue;
      double own[4];
      fl_mr_rec(a.z + ((size_t)(GRID ? node : t) * NR + k) * 4, own);
#pragma unroll
      for (int i = 0; i < D1; i++) {
        if (i < DIM && !pore) continue;
        const long j = (i < DIM ? DIM * t + i : DIM * nV + t) + k * n;
        a.s[j] = out[k][i];
        const double rv = a.r[j];
        vals[NV * k] += own[i] * out[k][i];
        vals[NV * k + 1] += rv * own[i];
        if constexpr (MAXN) {
          vals[NV * k + 2] = fmax(vals[NV * k + 2], fabs(rv));
          if (i < DIM) {  // the error norm reads the velocities (cfg.nhmg)
            vals[NV * k + 3] = fmax(vals[NV * k + 3], fabs(a.d[j]));
            vals[NV * k + 4] = fmax(vals[NV * k + 4], fabs(a.x[j]));
          }
        }
      }
    }
  }
  if (a.finish == FIN_NONE) return;
  bool ismax[NV * NR];
  double res[NV * NR];
#pragma unroll
  for (int k = 0; k < NV * NR; k++) ismax[k] = (k % NV) >= 2;
  if (grid_reduce<FL_NT, NV * NR>(vals, ismax, a.rc, blockIdx.x, res, sred) && threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NR; k++) {
      if (done[k]) continue;
      double s5[5] = {res[NV * k], res[NV * k + 1], 0.0, 0.0, 0.0};
      if constexpr (MAXN) { s5[2] = res[NV * k + 2]; s5[3] = res[NV * k + 3]; s5[4] = res[NV * k + 4]; }
      for (int m = 0; m < 5; m++) a.sc[k].red[m] = s5[m];
      mr_finish(a.finish, s5, a.sc + k, a.cfg);
    }
  }
}

}  // namespace chfem
