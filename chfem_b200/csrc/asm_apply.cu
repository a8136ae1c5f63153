// asm_apply.cu -- launches of the assembled-stencil block operator (stencil_asm.cuh) for every
// (dof per node, precision, block size) the block solver runs.
#include "asm_apply.h"
#include "device_cfg.h"
#include "stencil_asm.cuh"

namespace chfem {

namespace {
constexpr int ASM_TC = 8;  // columns of a tile
// The launched form: 32 x 8 columns, synchronous staging with an L2 bulk prefetch of the next step's
// planes, the table in shared memory, and registers capped so that two CTAs fit on an SM (FP64
// elastic planes of 19 doubles per node leave room for one: no cap there).
template <int ND, typename T, int NR>
constexpr auto asm_kernel = k_asm_apply<ND, T, NR, ASM_TC, ND == 1 ? 2 : 1, (ND == 3 && sizeof(T) == 8) ? 1 : 2>;
template <int ND, typename T, int NR>
size_t asm_smem() { return asm_smem_bytes<ND, T, NR, ASM_TC, ND == 1 ? 2 : 1>(); }
}  // namespace

template <int ND, typename T, int NR>
int asm_block_ctas(int R, int C, int L, int num_sms) {
  const size_t smem = asm_smem<ND, T, NR>();
  static PerDevice kept;
  const int per_sm = ctas_per_sm(kept, asm_kernel<ND, T, NR>, TE_TR * ASM_TC, smem);
  if (!per_sm) return 0;
  const long work = (long)((R + TE_TR - 1) / TE_TR) * ((C + ASM_TC - 1) / ASM_TC) * L;
  return (int)std::max(1L, std::min((long)per_sm * num_sms, work / TE_MIN_RUN));
}

template <int ND, typename T, int NR>
cudaError_t asm_block_launch(const BlkArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st) {
  asm_kernel<ND, T, NR><<<nb, dim3(TE_TR, ASM_TC), asm_smem<ND, T, NR>(), st>>>(a, tab);
  return cudaGetLastError();
}

template <int ND, typename T, int MODE>
int asm_te_ctas(int R, int C, int L, int num_sms) {
  static PerDevice kept;
  const int per_sm = ctas_per_sm(kept, k_te_apply<ND, T, MODE, true>, TE_NT, te_asm_smem_bytes<ND, T>());
  if (!per_sm) return 0;
  const long work = (long)((R + TE_TR - 1) / TE_TR) * ((C + TE_TC - 1) / TE_TC) * L;
  return (int)std::max(1L, std::min((long)per_sm * num_sms, work / TE_MIN_RUN));
}
template <int ND, typename T, int MODE>
cudaError_t asm_te_launch(const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st) {
  k_te_apply<ND, T, MODE, true><<<nb, dim3(TE_TR, TE_TC), te_asm_smem_bytes<ND, T>(), st>>>(a, tab);
  return cudaGetLastError();
}
#define CHFEM_ASM_TE_INSTANTIATE(ND, T, MODE)                 \
  template int asm_te_ctas<ND, T, MODE>(int, int, int, int); \
  template cudaError_t asm_te_launch<ND, T, MODE>(const TeArgs<ND, T>&, const T*, int, cudaStream_t);
CHFEM_ASM_TE_INSTANTIATE(1, float, TE_PLAIN)
CHFEM_ASM_TE_INSTANTIATE(1, float, TE_PCG)
CHFEM_ASM_TE_INSTANTIATE(1, float, TE_MR)
CHFEM_ASM_TE_INSTANTIATE(1, double, TE_PLAIN)
CHFEM_ASM_TE_INSTANTIATE(1, double, TE_PCG)
CHFEM_ASM_TE_INSTANTIATE(1, double, TE_MR)
CHFEM_ASM_TE_INSTANTIATE(3, float, TE_PLAIN)
CHFEM_ASM_TE_INSTANTIATE(3, float, TE_PCG)
CHFEM_ASM_TE_INSTANTIATE(3, float, TE_MR)
CHFEM_ASM_TE_INSTANTIATE(3, double, TE_PLAIN)
CHFEM_ASM_TE_INSTANTIATE(3, double, TE_PCG)
CHFEM_ASM_TE_INSTANTIATE(3, double, TE_MR)
CHFEM_ASM_TE_INSTANTIATE(1, float, TE_DIRDOT)
CHFEM_ASM_TE_INSTANTIATE(1, float, TE_UPD)
CHFEM_ASM_TE_INSTANTIATE(1, double, TE_DIRDOT)
CHFEM_ASM_TE_INSTANTIATE(1, double, TE_UPD)
CHFEM_ASM_TE_INSTANTIATE(3, float, TE_DIRDOT)
CHFEM_ASM_TE_INSTANTIATE(3, float, TE_UPD)
CHFEM_ASM_TE_INSTANTIATE(3, double, TE_DIRDOT)
CHFEM_ASM_TE_INSTANTIATE(3, double, TE_UPD)

#define CHFEM_ASM_INSTANTIATE(ND, T, NR)                                              \
  template int asm_block_ctas<ND, T, NR>(int, int, int, int);                    \
  template cudaError_t asm_block_launch<ND, T, NR>(const BlkArgs<ND, T>&, const T*, int, cudaStream_t);
CHFEM_ASM_INSTANTIATE(1, float, 3)
CHFEM_ASM_INSTANTIATE(1, double, 3)
CHFEM_ASM_INSTANTIATE(3, float, 6)
CHFEM_ASM_INSTANTIATE(3, double, 6)
CHFEM_ASM_INSTANTIATE(3, float, 3)
CHFEM_ASM_INSTANTIATE(3, double, 3)

}  // namespace chfem
