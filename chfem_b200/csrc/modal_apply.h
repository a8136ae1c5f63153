// modal_apply.h -- host entry of the passes in voxel modes (stencil_modal.cuh), compiled in their own
// translation units (modal_unit.cu, modal_apply.cu).
#pragma once
#include <cuda_runtime.h>
#include "stencil_te.cuh"

namespace chfem {

// The pass's table (md_table_words() values, FP64) from the dense element matrices of nmat <= 4
// materials (Kd[m][8 nd][8 nd]); false when a matrix is not that of an isotropic material on a
// cube (to 1e-12 of its largest entry), the structure the passes rely on, or its diagonal is not
// positive (a node inside such a phase has no inverse diagonal).
bool md_build_table(int nd, int nmat, const double* Kd, double* tab);
int md_table_words();
// whether the passes' 32-bit byte offsets in a layer hold a layer of R x C nodes
inline bool md_layer_fits(int nd, long R, long C) { return R * C * nd * 8 < 0xffff0000L; }

// CTAs of one pass (density: under a scalar density field, a.sdf) and one launch, with the
// contract of k_te_apply<ND, T, MODE>.
template <int ND, typename T, int MODE, bool DENS>
int md_pass_ctas(int R, int C, int L, int num_sms);
template <int ND, typename T, int MODE, bool DENS>
cudaError_t md_pass_launch(const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st);
template <int ND, typename T, int MODE>
int md_ctas(bool density, int R, int C, int L, int num_sms) {
  return density ? md_pass_ctas<ND, T, MODE, true>(R, C, L, num_sms) : md_pass_ctas<ND, T, MODE, false>(R, C, L, num_sms);
}
template <int ND, typename T, int MODE>
cudaError_t md_launch(const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st) {
  return a.sdf ? md_pass_launch<ND, T, MODE, true>(a, tab, nb, st) : md_pass_launch<ND, T, MODE, false>(a, tab, nb, st);
}

// The block PCG operator pass on nr right-hand sides (contract of k_blk_apply); a: the fields of
// the first of them (in0 = r, in1 = d_old, vout = d_new, y = q), n unknowns apart.
template <int ND, typename T>
int md_block_ctas(int nr, int R, int C, int L, int num_sms);
template <int ND, typename T>
cudaError_t md_block_launch(int nr, long n, const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st);

// The pointwise PCG pass (modal_point.cuh) on nr right-hand sides, n unknowns apart; parity: which
// pass of a pair (x is updated in the second), norms: the stopping test reads max-norms (x is
// updated in every pass).
template <typename T>
struct MdPw;
int md_point_ctas(long n, int num_sms);
template <int ND, typename T>
cudaError_t md_point_single(const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st);
template <int ND, typename T>
cudaError_t md_point_block(int nr, const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st);
template <int ND, typename T>
cudaError_t md_point_launch(int nr, const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  return nr == 1 ? md_point_single<ND, T>(a, parity, norms, nb, st) : md_point_block<ND, T>(nr, a, parity, norms, nb, st);
}

}  // namespace chfem
