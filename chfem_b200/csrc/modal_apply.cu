// modal_apply.cu -- the table of the passes in voxel modes (stencil_modal.cuh); their launches are in
// modal_unit.cu.
#include <algorithm>
#include <cmath>
#include <vector>
#include "modal_apply.h"
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

// CTAs of 256 threads: 4 per SM keep enough 16-byte loads in flight for the memory's latency and
// the partials that the last CTA sums few.
int md_point_ctas(long n, int num_sms) { return (int)std::max(1L, std::min(4L * num_sms, (n / 2 + MP_NT - 1) / MP_NT)); }

}  // namespace chfem
