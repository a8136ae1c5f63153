// modal_unit.cu -- launches of the passes in voxel modes (stencil_modal.cuh, modal_point.cuh) for MD_ND
// unknowns per node and fields of type MD_T, one part of them at a time: MD_PASS the operator passes
// of one right-hand side, MD_DENSITY the same under a scalar density field, MD_BLOCK the passes of a
// block, MD_POINT the pointwise pass of one right-hand side.  Each combination is compiled to a
// module of its own, of which a process runs two or three: the first launch of any kernel loads its
// whole module, which took 23 ms in every process with all of them in one, against 1.5 to 2 ms (the
// first operator apply of thermal 64^3 and elastic 48^3; the passes before took 1.9 and 5.9).
#include <algorithm>
#include "modal_apply.h"
#include "device_cfg.h"
#include "modal_point.cuh"

namespace chfem {

#if !defined(MD_POINT)
namespace {
// CTAs per SM the registers are capped for: as many as fit without spills (stencil_modal.cuh).
template <int ND, typename V>
constexpr int md_minb = ND == 1 ? (sizeof(V) == 8 ? 3 : 4) : (sizeof(V) == 8 ? 1 : 2);
template <int ND, typename V, int MODE, bool BLK, bool DENS>
constexpr auto md_kernel = k_modal_apply<ND, V, MODE, md_minb<ND, V>, BLK, DENS>;

// CTAs of one pass: as many as fit on the GPU at once, but 8 layers of a tile each at least -- a CTA's
// fixed cost (table, first planes, its share of the reduction) outweighs fewer -- while that leaves
// the SMs a CTA each, or two in the passes of (P)MINRES and the 3-vector PCG (whose layers wait on
// more loads) and in models of more tiles than SMs (whose runs would cross tiles and restage planes).
// Thermal FP64, us between events around a launch, one per SM against two: PCG pass 64^3 14.6 and
// 14.7 (three: 15.3), 4 x 256 x 256 18.8 and 14.7; (P)MINRES pass 64^3 22.8 and 21.4, 4 x 256 x 256
// 28.3 and 22.0.  The 3-vector PCG, both passes: 64^3 29.2 and 27.0 us an iteration.
template <int ND, typename V, int MODE, bool BLK, bool DENS>
int ctas_of(int groups, int R, int C, int L, int num_sms) {
  const size_t smem = md_smem_bytes<ND, V>();
  static PerDevice kept;
  const int per_sm = ctas_per_sm(kept, md_kernel<ND, V, MODE, BLK, DENS>, MD_NT, smem);
  if (!per_sm) return 0;
  const long tiles = (long)groups * ((R + TE_TR - 1) / TE_TR) * ((C + MD_TC - 1) / MD_TC), work = tiles * L;
  constexpr long least = MODE == TE_MR || MODE == TE_DIRDOT || MODE == TE_UPD ? 2 : 1;
  const long want = std::min(work, std::max({least * num_sms, std::min(tiles, 2L * num_sms), work / 8}));
  return (int)std::max((long)groups, std::min((long)per_sm * num_sms, want));
}
template <int ND, typename V, int MODE, bool BLK, bool DENS>
cudaError_t launch(const MdArgs<ND, typename MdV<V>::T>& a, int nb, cudaStream_t st) {
  md_kernel<ND, V, MODE, BLK, DENS><<<nb, MD_NT, md_smem_bytes<ND, V>(), st>>>(a);
  return cudaGetLastError();
}
}  // namespace

#endif

#if defined(MD_PASS) || defined(MD_DENSITY)
#ifdef MD_DENSITY
constexpr bool WITH_DENSITY = true;
#else
constexpr bool WITH_DENSITY = false;
#endif
template <int ND, typename T, int MODE, bool DENS>
int md_pass_ctas(int R, int C, int L, int num_sms) {
  return ctas_of<ND, T, MODE, false, DENS>(1, R, C, L, num_sms);
}
template <int ND, typename T, int MODE, bool DENS>
cudaError_t md_pass_launch(const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st) {
  return launch<ND, T, MODE, false, DENS>(MdArgs<ND, T>{a, tab, 0, 1}, nb, st);
}
#define CHFEM_MD_INSTANTIATE(MODE)                                                 \
  template int md_pass_ctas<MD_ND, MD_T, MODE, WITH_DENSITY>(int, int, int, int); \
  template cudaError_t md_pass_launch<MD_ND, MD_T, MODE, WITH_DENSITY>(const TeArgs<MD_ND, MD_T>&, const MD_T*, int, cudaStream_t);
CHFEM_MD_INSTANTIATE(TE_PLAIN)
CHFEM_MD_INSTANTIATE(TE_PCG)
CHFEM_MD_INSTANTIATE(TE_MR)
CHFEM_MD_INSTANTIATE(TE_DIRDOT)
CHFEM_MD_INSTANTIATE(TE_UPD)
#endif

#ifdef MD_BLOCK
// A pair of right-hand sides per CTA where their number is even and the fields are FP32 (packed
// FP32 arithmetic), else one.
template <int ND, typename T>
int md_block_ctas(int nr, int R, int C, int L, int num_sms) {
  if constexpr (sizeof(T) == 4) {
    if (nr % 2 == 0) return ctas_of<ND, float2, TE_PCG, true, false>(nr / 2, R, C, L, num_sms);
  }
  return ctas_of<ND, T, TE_PCG, true, false>(nr, R, C, L, num_sms);
}
template <int ND, typename T>
cudaError_t md_block_launch(int nr, long n, const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st) {
  const MdArgs<ND, T> ma{a, tab, n, nr};
  if constexpr (sizeof(T) == 4) {
    if (nr % 2 == 0) return launch<ND, float2, TE_PCG, true, false>(ma, nb, st);
  }
  return launch<ND, T, TE_PCG, true, false>(ma, nb, st);
}
template int md_block_ctas<MD_ND, MD_T>(int, int, int, int, int);
template cudaError_t md_block_launch<MD_ND, MD_T>(int, long, const TeArgs<MD_ND, MD_T>&, const MD_T*, int, cudaStream_t);
#endif

#if defined(MD_BLOCK) || defined(MD_POINT)
namespace {
template <int ND, typename T, int NR, int VW>
void point(const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  if (norms) k_md_point<ND, T, NR, 2, VW><<<nb, MP_NT, 0, st>>>(a);
  else if (parity) k_md_point<ND, T, NR, 1, VW><<<nb, MP_NT, 0, st>>>(a);
  else k_md_point<ND, T, NR, 0, VW><<<nb, MP_NT, 0, st>>>(a);
}
// The widest words that all of the block's vectors start on; one right-hand side always starts on
// 16 bytes.
template <int ND, typename T, int NR>
void point_width(const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  constexpr int FULL = 16 / (int)sizeof(T);
  if constexpr (NR == 1) point<ND, T, NR, FULL>(a, parity, norms, nb, st);
  else if (a.n % FULL == 0) point<ND, T, NR, FULL>(a, parity, norms, nb, st);
  else if (FULL == 4 && a.n % 2 == 0) point<ND, T, NR, 2>(a, parity, norms, nb, st);
  else point<ND, T, NR, 1>(a, parity, norms, nb, st);
}
}  // namespace
#ifdef MD_POINT
template <int ND, typename T>
cudaError_t md_point_single(const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  point_width<ND, T, 1>(a, parity, norms, nb, st);
  return cudaGetLastError();
}
template cudaError_t md_point_single<MD_ND, MD_T>(const MdPw<MD_T>&, int, bool, int, cudaStream_t);
#else
template <int ND, typename T>
cudaError_t md_point_block(int nr, const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  if (nr == 3) point_width<ND, T, 3>(a, parity, norms, nb, st);
  else if constexpr (ND == 3) point_width<ND, T, 6>(a, parity, norms, nb, st);
  return cudaGetLastError();
}
template cudaError_t md_point_block<MD_ND, MD_T>(int, const MdPw<MD_T>&, int, bool, int, cudaStream_t);
#endif
#endif

}  // namespace chfem
