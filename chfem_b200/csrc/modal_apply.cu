// modal_apply.cu -- launches of the operator passes in voxel modes (stencil_modal.cuh), and their
// table.
#include <algorithm>
#include <cmath>
#include <vector>
#include "modal_apply.h"
#include "device_cfg.h"
#include "stencil_modal.cuh"
#include "modal_point.cuh"

namespace chfem {

int md_table_words() { return MD_WORDS; }

bool md_build_table(int nd, int nmat, const double* Kd, double* tab) {
  if (nmat < 1 || nmat > 4) return false;
  const int ED = 8 * nd;
  for (int i = 0; i < MD_WORDS; i++) tab[i] = 0.0;
  // H: mode m (bit 0 rows, bit 1 columns, bit 2 layers) of local node k
  double H[8][8];
  for (int m = 0; m < 8; m++)
    for (int k = 0; k < 8; k++) {
      double s = 1.0;
      if (m & 1) s *= drow(k) == 0 ? -1.0 : 1.0;
      if (m & 2) s *= dcol(k) ? 1.0 : -1.0;
      if (m & 4) s *= dlay(k) ? -1.0 : 1.0;
      H[m][k] = s;
    }
  constexpr int Y = 1, X = 2, Z = 4;
  double diag[4] = {0.0, 0.0, 0.0, 0.0};
  std::vector<double> M((size_t)ED * ED), G((size_t)ED * ED), want((size_t)ED * ED);
  for (int mat = 0; mat < nmat; mat++) {
    const double* K = Kd + (size_t)mat * ED * ED;
    double big = 0.0;
    for (int i = 0; i < ED * ED; i++) big = std::max(big, std::fabs(K[i]));
    const double tol = 1e-12 * big;
    diag[mat] = K[0];
    if (!(diag[mat] > 0.0)) return false;
    for (int i = 0; i < ED; i++)
      if (!(std::fabs(K[i * ED + i] - diag[mat]) <= tol)) return false;
    // M = H K H^T / 64 per component pair
    for (int m = 0; m < 8; m++)
      for (int ci = 0; ci < nd; ci++)
        for (int j = 0; j < ED; j++) {
          double s = 0.0;
          for (int k = 0; k < 8; k++) s += H[m][k] * K[(k * nd + ci) * ED + j];
          G[(size_t)(m * nd + ci) * ED + j] = s;
        }
    for (int i = 0; i < ED; i++)
      for (int m = 0; m < 8; m++)
        for (int cj = 0; cj < nd; cj++) {
          double s = 0.0;
          for (int k = 0; k < 8; k++) s += G[(size_t)i * ED + k * nd + cj] * H[m][k];
          M[(size_t)i * ED + m * nd + cj] = s / 64.0;
        }
    auto at = [&](int m, int c) { return m * nd + c; };
    std::fill(want.begin(), want.end(), 0.0);
    auto set = [&](int a, int b, double v) { want[(size_t)a * ED + b] = v; want[(size_t)b * ED + a] = v; };
    double lam, mu = 0.0;
    if (nd == 1) {
      lam = M[(size_t)X * ED + X];
      for (int m : {X, Y, Z}) set(m, m, lam);
      for (int m : {X | Y, X | Z, Y | Z}) set(m, m, lam * 2.0 / 3.0);
      set(7, 7, lam / 3.0);
    } else {
      lam = M[(size_t)at(X, 0) * ED + at(Y, 1)];
      mu = M[(size_t)at(Y, 0) * ED + at(X, 1)];
      const int nrm[3] = {at(X, 0), at(Y, 1), at(Z, 2)}, tw[3] = {at(Y | Z, 0), at(X | Z, 1), at(X | Y, 2)};
      const int sh[3][2] = {{at(Y, 0), at(X, 1)}, {at(Z, 0), at(X, 2)}, {at(Z, 1), at(Y, 2)}};
      const int pr[3][2] = {{at(X | Z, 0), at(Y | Z, 1)}, {at(X | Y, 0), at(Y | Z, 2)}, {at(X | Y, 1), at(X | Z, 2)}};
      for (int a = 0; a < 3; a++) {
        for (int b = 0; b < 3; b++) {
          set(nrm[a], nrm[b], a == b ? lam + 2.0 * mu : lam);
          set(tw[a], tw[b], a == b ? mu * 2.0 / 3.0 : mu / 3.0);
        }
        set(sh[a][0], sh[a][0], mu); set(sh[a][1], sh[a][1], mu); set(sh[a][0], sh[a][1], mu);
        set(pr[a][0], pr[a][0], lam / 3.0 + mu); set(pr[a][1], pr[a][1], lam / 3.0 + mu); set(pr[a][0], pr[a][1], lam / 3.0);
        set(at(7, a), at(7, a), (lam + 4.0 * mu) / 9.0);
      }
    }
    for (size_t i = 0; i < want.size(); i++)
      if (!(std::fabs(M[i] - want[i]) <= tol)) return false;
    tab[MD_MAT + 2 * mat] = lam;
    tab[MD_MAT + 2 * mat + 1] = mu;
  }
  for (int n3 = 0; n3 <= 8; n3++)
    for (int n2 = 0; n2 + n3 <= 8; n2++)
      for (int n1 = 0; n1 + n2 + n3 <= 8; n1++) {
        const int n0 = 8 - n1 - n2 - n3;
        const double d = n0 * diag[0] + n1 * diag[1] + n2 * diag[2] + n3 * diag[3];
        tab[n1 + 9 * n2 + 81 * n3] = d != 0.0 ? 1.0 / d : 0.0;  // 0: counts of materials the model lacks
      }
  return true;
}

namespace {
// CTAs per SM the registers are capped for: as many as fit without spills (stencil_modal.cuh).
template <int ND, typename V>
constexpr int md_minb = ND == 1 ? (sizeof(V) == 8 ? 3 : 4) : (sizeof(V) == 8 ? 1 : 2);
template <int ND, typename V, int MODE, bool BLK, bool DENS>
constexpr auto md_kernel = k_modal_apply<ND, V, MODE, md_minb<ND, V>, BLK, DENS>;

// CTAs of one pass: as many as fit on the GPU at once, but 8 layers of a tile each at least while
// that leaves one per SM -- a CTA's fixed cost (table, first planes, its share of the reduction)
// outweighs fewer layers: thermal 64^3 FP64 14.8 us at 148 CTAs, 18.0 at 444.
template <int ND, typename V, int MODE, bool BLK, bool DENS>
int ctas_of(int groups, int R, int C, int L, int num_sms) {
  const size_t smem = md_smem_bytes<ND, V>();
  static PerDevice kept;
  const int per_sm = ctas_per_sm(kept, md_kernel<ND, V, MODE, BLK, DENS>, MD_NT, smem);
  if (!per_sm) return 0;
  const long work = (long)groups * ((R + TE_TR - 1) / TE_TR) * ((C + MD_TC - 1) / MD_TC) * L;
  const long want = std::min(work, std::max((long)num_sms, work / 8));
  return (int)std::max((long)groups, std::min((long)per_sm * num_sms, want));
}
template <int ND, typename V, int MODE, bool BLK, bool DENS>
cudaError_t launch(const MdArgs<ND, typename MdV<V>::T>& a, int nb, cudaStream_t st) {
  md_kernel<ND, V, MODE, BLK, DENS><<<nb, MD_NT, md_smem_bytes<ND, V>(), st>>>(a);
  return cudaGetLastError();
}
}  // namespace

template <int ND, typename T, int MODE>
int md_ctas(bool density, int R, int C, int L, int num_sms) {
  return density ? ctas_of<ND, T, MODE, false, true>(1, R, C, L, num_sms) : ctas_of<ND, T, MODE, false, false>(1, R, C, L, num_sms);
}
template <int ND, typename T, int MODE>
cudaError_t md_launch(const TeArgs<ND, T>& a, const T* tab, int nb, cudaStream_t st) {
  const MdArgs<ND, T> ma{a, tab, 0, 1};
  return a.sdf ? launch<ND, T, MODE, false, true>(ma, nb, st) : launch<ND, T, MODE, false, false>(ma, nb, st);
}

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

#define CHFEM_MD_INSTANTIATE(ND, T, MODE)                 \
  template int md_ctas<ND, T, MODE>(bool, int, int, int, int); \
  template cudaError_t md_launch<ND, T, MODE>(const TeArgs<ND, T>&, const T*, int, cudaStream_t);
#define CHFEM_MD_MODES(ND, T)           \
  CHFEM_MD_INSTANTIATE(ND, T, TE_PLAIN) \
  CHFEM_MD_INSTANTIATE(ND, T, TE_PCG)   \
  CHFEM_MD_INSTANTIATE(ND, T, TE_MR)    \
  CHFEM_MD_INSTANTIATE(ND, T, TE_DIRDOT) \
  CHFEM_MD_INSTANTIATE(ND, T, TE_UPD)
CHFEM_MD_MODES(1, float)
CHFEM_MD_MODES(1, double)
CHFEM_MD_MODES(3, float)
CHFEM_MD_MODES(3, double)
#define CHFEM_MD_BLOCK(ND, T)                            \
  template int md_block_ctas<ND, T>(int, int, int, int, int); \
  template cudaError_t md_block_launch<ND, T>(int, long, const TeArgs<ND, T>&, const T*, int, cudaStream_t);
CHFEM_MD_BLOCK(1, float)
CHFEM_MD_BLOCK(1, double)
CHFEM_MD_BLOCK(3, float)
CHFEM_MD_BLOCK(3, double)

// CTAs of 256 threads: 4 per SM keep enough 16-byte loads in flight for the memory's latency and
// the partials that the last CTA sums few.
int md_point_ctas(long n, int num_sms) { return (int)std::max(1L, std::min(4L * num_sms, (n / 2 + MP_NT - 1) / MP_NT)); }

namespace {
template <int ND, typename T, int NR, int VW>
void point(const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  if (norms) k_md_point<ND, T, NR, 2, VW><<<nb, MP_NT, 0, st>>>(a);
  else if (parity) k_md_point<ND, T, NR, 1, VW><<<nb, MP_NT, 0, st>>>(a);
  else k_md_point<ND, T, NR, 0, VW><<<nb, MP_NT, 0, st>>>(a);
}
template <int ND, typename T, int NR>
void point_width(const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  constexpr int FULL = 16 / (int)sizeof(T);
  if (NR == 1 || a.n % FULL == 0) point<ND, T, NR, FULL>(a, parity, norms, nb, st);
  else if (FULL == 4 && a.n % 2 == 0) point<ND, T, NR, 2>(a, parity, norms, nb, st);
  else point<ND, T, NR, 1>(a, parity, norms, nb, st);
}
}  // namespace
template <int ND, typename T>
cudaError_t md_point_launch(int nr, const MdPw<T>& a, int parity, bool norms, int nb, cudaStream_t st) {
  if (nr == 1) point_width<ND, T, 1>(a, parity, norms, nb, st);
  else if (nr == 3) point_width<ND, T, 3>(a, parity, norms, nb, st);
  else if constexpr (ND == 3) point_width<ND, T, 6>(a, parity, norms, nb, st);
  return cudaGetLastError();
}
template cudaError_t md_point_launch<1, float>(int, const MdPw<float>&, int, bool, int, cudaStream_t);
template cudaError_t md_point_launch<1, double>(int, const MdPw<double>&, int, bool, int, cudaStream_t);
template cudaError_t md_point_launch<3, float>(int, const MdPw<float>&, int, bool, int, cudaStream_t);
template cudaError_t md_point_launch<3, double>(int, const MdPw<double>&, int, bool, int, cudaStream_t);

}  // namespace chfem
