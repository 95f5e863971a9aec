// screen_check.cpp -- TEST INFRASTRUCTURE ONLY: the constants that the screens
// of the int8 kernels take from a phenotype's limb columns.
#include <cmath>
#include <cstring>

#include "../../supergwas_b200/csrc/params.hpp"

// r2_cand: the emit cut; ref: the refinement threshold (r2).  loss: bounds of
// limb_loss (u, y).  d: the prepared columns, k + 1 of n values.  Returns 0, or 1 where the structure is refused.
extern "C" int screen_constants(const double* U, int n, int k, const double* y, double r2_cand, double ref,
                                double* loss, double* need, int* on, double* d) {
  kg::Prepared p;
  kg::LimbCols L;
  if (!kg::prepare(U, n, k, y, p).empty() || !kg::make_limbs(p, nullptr, n, 3, 5, 128, L).empty()) return 1;
  kg::EpiParams P;
  std::memset(&P, 0, sizeof(P));
  P.n = n;
  P.k = k;
  P.b = p.b;
  P.kappa = p.kappa;
  P.yyM = p.yyM;
  P.ynorm = p.ynorm;
  P.r2_cand = r2_cand;
  P.r2_ref = ref;
  P.refine = 1;
  for (int j = 0; j < k; ++j) P.a[j] = p.a[j], P.g[j] = p.g[j];
  kg::LimbMap LM;
  std::memset(&LM, 0, sizeof(LM));
  for (int j = 0; j <= k; ++j) LM.scale[j] = L.scale[j];
  kg::LimbLoss B;
  kg::limb_loss(p, LM.scale, B);
  kg::set_refine_need(P, B);
  kg::set_screen(P, LM, p.drop0, B);
  loss[0] = B.u;
  loss[1] = B.y;
  *need = P.r2_need;
  *on = P.S.on;
  std::memcpy(d, p.d.data(), p.d.size() * sizeof(double));
  return 0;
}
