// prep.cpp -- see prep.hpp for the algebra.
#include "prep.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace kg {

typedef long double ld;

std::string prepare(const double* U, int n, int k, const double* y, Prepared& P) {
  if (n <= 0) return "n must be positive";
  if (k < 0 || k > KMAX) return "k (U.bin columns) must be in [0, " + std::to_string(KMAX) + "]";
  if (!y) return "y is NULL";
  if (k > 0 && !U) return "U is NULL";
  for (int i = 0; i < n; ++i)
    if (!std::isfinite(y[i])) return "phenotype value is not finite";
  for (size_t i = 0; i < (size_t)n * k; ++i)
    if (!std::isfinite(U[i])) return "U.bin value is not finite";

  P = Prepared();
  P.n = n;
  P.k = k;
  // U^T y and yyM (src/kgwas_utils.hpp:151-153), ynorm of y - mean(y)
  std::vector<ld> Uy(k);
  ld yy = 0, ysum = 0;
  for (int i = 0; i < n; ++i) { yy += (ld)y[i] * y[i]; ysum += y[i]; }
  ld uyy = 0;
  for (int j = 0; j < k; ++j) {
    ld s = 0;
    for (int i = 0; i < n; ++i) s += (ld)U[(size_t)j * n + i] * y[i];
    Uy[j] = s;
    uyy += s * s;
  }
  P.yyM = (double)(yy - uyy);
  const ld ymean = ysum / n;
  P.ymean = (double)ymean;
  ld yc2 = 0;
  for (int i = 0; i < n; ++i) { ld t = (ld)y[i] - ymean; yc2 += t * t; }
  P.ynorm = (double)std::sqrt(yc2);

  // Householder H with H e0 = w/||w||, w = U^T 1; Q = U H.
  std::vector<ld> Q((size_t)n * (k > 0 ? k : 1), 0);
  for (size_t i = 0; i < (size_t)n * k; ++i) Q[i] = U[i];
  std::vector<ld> w(k, 0);
  ld wn2 = 0;
  for (int j = 0; j < k; ++j) {
    ld s = 0;
    for (int i = 0; i < n; ++i) s += U[(size_t)j * n + i];
    w[j] = s;
    wn2 += s * s;
  }
  std::vector<ld> Hm((size_t)k * k, 0);  // H, row-major
  for (int j = 0; j < k; ++j) Hm[(size_t)j * k + j] = 1;
  if (k > 0 && wn2 > 0) {
    const ld wn = std::sqrt(wn2);
    std::vector<ld> v(k);
    ld vv = 0;
    for (int j = 0; j < k; ++j) { v[j] = w[j] / wn - (j == 0 ? 1 : 0); vv += v[j] * v[j]; }
    if (vv > 1e-30L) {
      for (int r = 0; r < k; ++r)
        for (int c = 0; c < k; ++c) Hm[(size_t)r * k + c] -= 2 * v[r] * v[c] / vv;
      // Q = U H: Q[:, c] = sum_r U[:, r] H[r, c]
      for (int c = 0; c < k; ++c)
        for (int i = 0; i < n; ++i) {
          ld s = 0;
          for (int r = 0; r < k; ++r) s += (ld)U[(size_t)r * n + i] * Hm[(size_t)r * k + c];
          Q[(size_t)c * n + i] = s;
        }
    }
  }
  // g = Q^T y = H U^T y (H symmetric)
  P.a.assign(k, 0.0);
  P.g.assign(k, 0.0);
  std::vector<ld> gl(k, 0), al(k, 0);
  for (int c = 0; c < k; ++c) {
    ld s = 0;
    for (int r = 0; r < k; ++r) s += Hm[(size_t)r * k + c] * Uy[r];
    gl[c] = s;
    P.g[c] = (double)s;
  }
  P.d.assign((size_t)(k + 1) * n, 0.0);
  for (int j = 0; j < k; ++j) {
    ld s = 0;
    for (int i = 0; i < n; ++i) s += Q[(size_t)j * n + i];
    al[j] = s / n;
    P.a[j] = (double)al[j];
    for (int i = 0; i < n; ++i) P.d[(size_t)j * n + i] = (double)(Q[(size_t)j * n + i] - al[j]);
  }
  // y' = y - U (U^T y); b = mean(y'); d_y = y' - b
  std::vector<ld> yp(n);
  ld ps = 0;
  for (int i = 0; i < n; ++i) {
    ld s = y[i];
    for (int j = 0; j < k; ++j) s -= (ld)U[(size_t)j * n + i] * Uy[j];
    yp[i] = s;
    ps += s;
  }
  const ld bl = ps / n;
  P.b = (double)bl;
  for (int i = 0; i < n; ++i) P.d[(size_t)k * n + i] = (double)(yp[i] - bl);
  ld kap = bl - ymean;
  for (int j = 0; j < k; ++j) kap += al[j] * gl[j];
  P.kappa = (double)kap;
  // Column 0's centred part is rounding noise when 1 lies in span(U).
  if (k > 0) {
    double mx = 0;
    for (int i = 0; i < n; ++i) mx = std::max(mx, std::fabs(P.d[i]));
    P.drop0 = (mx <= 1e-13 * std::fabs(P.a[0]));
  }
  return "";
}

// Balanced signed-digit decomposition of V into L base-256 digits in [-128,127].
static void digits(int64_t V, int L, int8_t* out) {
  for (int l = L - 1; l >= 0; --l) {
    int64_t r = ((V % 256) + 256) % 256;  // 0..255
    int64_t dgt = r >= 128 ? r - 256 : r;
    out[l] = (int8_t)dgt;
    V = (V - dgt) / 256;
  }
}

std::string make_limbs(const Prepared& p, const int* pos, int n_row, int limbs_u, int limbs_y, int kquant,
                       LimbCols& L) {
  if (limbs_u < 1 || limbs_u > 4 || limbs_y < 1 || limbs_y > 5) return "limbs must be in [1, 4] for U and [1, 5] for y'";
  const int n = p.n, k = p.k;
  if (n_row < n) return "rows hold fewer samples than the overlap";
  L = LimbCols();
  L.Kpad = ((n_row + kquant - 1) / kquant) * kquant;
  // column order: [count, y' limbs, U column 0 (unless dropped), U columns 1..k-1]
  int col = 0;
  L.count_col = col++;
  L.first[k] = col;
  L.nl[k] = limbs_y;
  L.scale[k] = 0.0;
  col += limbs_y;
  for (int j = 0; j < k; ++j) {
    const bool skip = (j == 0 && p.drop0);
    const int nl = skip ? 0 : limbs_u;
    L.first[j] = col;
    L.nl[j] = nl;
    L.scale[j] = 0.0;
    col += nl;
  }
  const int used = col;
  int N = ((used + 15) / 16) * 16;
  if (N < 16) N = 16;
  if (N > 256) return "too many contraction columns for one MMA (" + std::to_string(used) + " > 256)";
  L.N = N;
  L.vals.assign((size_t)N * L.Kpad, 0);
  auto at = [&](int i) { return pos ? pos[i] : i; };
  for (int i = 0; i < n; ++i) L.vals[(size_t)L.count_col * L.Kpad + at(i)] = 1;
  std::vector<int8_t> dg(8);
  for (int j = 0; j <= k; ++j) {
    const int nl = L.nl[j];
    if (nl == 0) continue;
    const double* v = &p.d[(size_t)j * n];
    double mx = 0;
    for (int i = 0; i < n; ++i) mx = std::max(mx, std::fabs(v[i]));
    // half the largest magnitude representable with a top digit in
    // [-127, 127]: the TMEM kernel multiplies half of the samples as 64 x
    // against the digits of -2 V (make_b_image_ts), which must fit too
    const double lim = 127.0 * std::ldexp(1.0, 8 * (nl - 1) - 1);
    int s = 0;
    if (mx > 0) {
      int e;
      std::frexp(lim / mx, &e);   // lim/mx in [2^(e-1), 2^e)
      s = e - 1;                  // mx * 2^s <= lim
    }
    L.scale[j] = std::ldexp(1.0, -s);
    for (int i = 0; i < n; ++i) {
      const int64_t V = (int64_t)std::llround(std::ldexp(v[i], s));
      digits(V, nl, dg.data());
      for (int l = 0; l < nl; ++l) L.vals[(size_t)(L.first[j] + l) * L.Kpad + at(i)] = dg[l];
    }
  }
  return "";
}

void put_b_image_ts(const LimbCols& L, int col0, int N, std::vector<int8_t>& img) {
  // Limb digits of -2 V for every sample, column by column (V = the value a
  // logical column's digits encode; the count column holds V = 1).
  std::vector<int8_t> neg2((size_t)L.N * L.Kpad, 0);
  std::vector<int8_t> dg(8);
  auto regroup = [&](int first, int nl) {
    for (int i = 0; i < L.Kpad; ++i) {
      int64_t V = 0;
      for (int l = 0; l < nl; ++l) V = V * 256 + L.vals[(size_t)(first + l) * L.Kpad + i];
      digits(-2 * V, nl, dg.data());
      for (int l = 0; l < nl; ++l) neg2[(size_t)(first + l) * L.Kpad + i] = dg[l];
    }
  };
  regroup(L.count_col, 1);
  for (int j = 0; j <= KMAX; ++j)
    if (L.nl[j] > 0 && L.first[j] > 0 && L.first[j] + L.nl[j] <= L.N) regroup(L.first[j], L.nl[j]);
  for (int kap = 0; kap < L.Kpad; ++kap) {
    // TMEM column c of a 128-sample stage holds K = 4c..4c+3.  The unpack
    // (unpack_stage in device.cuh) writes, for 32-bit word q of the stage and
    // jj = 0..7, column 8q+jj = (word << 2*(jj/2)) & (jj even ? 0x80808080 :
    // 0x40404040): byte t of it is sample 32q + 8t + 7 - jj, as -128 x (jj
    // even) or 64 x (jj odd).  Odd columns therefore take the digits of -2 V.
    const int a = kap / 128, w = kap % 128, c = w / 4, t = w % 4, q = c / 8, jj = c % 8;
    const int i = 128 * a + 32 * q + 8 * t + 7 - jj;
    const std::vector<int8_t>& src = (jj & 1) ? neg2 : L.vals;
    for (int col = 0; col < L.N; ++col) {
      const int cc = col0 + col;
      const size_t off = (size_t)(kap / 16) * (N * 16) + (size_t)(cc / 8) * 128 + (size_t)(cc % 8) * 16 + kap % 16;
      img[off] = src[(size_t)col * L.Kpad + i];
    }
  }
}

void make_b_image_ts(const LimbCols& L, std::vector<int8_t>& img) {
  img.assign((size_t)L.Kpad * L.N, 0);
  put_b_image_ts(L, 0, L.N, img);
}

void make_b_image(const LimbCols& L, int KC, std::vector<int8_t>& img) {
  const int N = L.N, nchunk = L.Kpad / KC;
  img.assign((size_t)L.Kpad * N, 0);
  for (int q = 0; q < nchunk; ++q)
    for (int k16 = 0; k16 < KC / 16; ++k16)
      for (int col = 0; col < N; ++col)
        for (int kk = 0; kk < 16; ++kk) {
          const int i = q * KC + k16 * 16 + kk;
          const size_t off = (size_t)q * KC * N + (size_t)k16 * (N * 16) + (size_t)(col / 8) * 128 +
                             (size_t)(col % 8) * 16 + kk;
          img[off] = L.vals[(size_t)col * L.Kpad + i];
        }
}

// ------------------------------------------------------------ 4-bit screen
// Nearest integer (|t| < 2^22), in two additions that vectorise.
static inline float near_int(float t) { return (t + 12582912.0f) - 12582912.0f; }
// Nearest e2m1 value of t (|t| above 6 becomes 6), without branches.
static inline float e2m1_round(float t) {
  const float a = std::min(std::fabs(t), 6.0f);
  const float h = near_int(a * 2.0f) * 0.5f, w = near_int(a), d = near_int(a * 0.5f) * 2.0f;
  const float ge2 = a >= 2.0f ? 1.0f : 0.0f, ge4 = a >= 4.0f ? 1.0f : 0.0f;
  return std::copysign(h + (w - h) * ge2 + (d - w) * ge4, t);
}
static inline uint8_t e2m1_code(float v) {
  const int h = (int)(std::fabs(v) * 2.0f);  // 0 1 2 3 4 6 8 12
  const int c = h <= 4 ? h : h == 6 ? 5 : h == 8 ? 6 : 7;
  return (uint8_t)(c | (v < 0 ? 8 : 0));
}

// Moves codes of the last limb (scale s) to a neighbouring value, where that adds
// little to the residual r, until the residual's sum is as close to zero as one
// such step allows.  A row of frequency near one meets the sum: the rest of the
// bound shrinks with ||x - mean(x)||, c |sum r| / n does not.
static void fs_balance(std::vector<double>& r, const int* pos, uint8_t* code, double s) {
  static const float val[8] = {0.0f, 0.5f, 1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f};
  const int n = (int)r.size();
  double D = 0;
  for (double v : r) D += v;
  // in units of s; passes over the entries, the nearest to a tie first
  for (float most : {0.02f, 0.1f, 0.3f, 1.0f, 8.0f}) {
    for (int i = 0; i < n && std::fabs(D) > 0.25 * s; ++i) {
      const int dir = D > 0 ? 1 : -1;  // a positive sum: larger limbs
      uint8_t& c = code[pos ? pos[i] : i];
      const int at = (c & 8) ? -(c & 7) : (c & 7), to = at + dir;
      if (to > 7 || to < -7) continue;
      const float q = at < 0 ? -val[-at] : val[at], q2 = to < 0 ? -val[-to] : val[to];
      const double step = s * (double)(q2 - q), moved = r[i] - step;
      if (!(moved * moved - r[i] * r[i] <= most * s * s) || std::fabs(D - step) >= std::fabs(D)) continue;
      D -= step;
      r[i] = moved;
      c = (uint8_t)(to < 0 ? 8 | -to : to);
    }
  }
}

// The limbs of column r (n values): the codes (limb l to code + l * stride) and
// the scales; r keeps what they leave out.  The last two limbs take the nearest
// e2m1 values, with the scale, of a few below the one that represents the
// largest value, that leaves the least.  The limbs before it keep to the
// integers up to 4, whose even spacing leaves the next limb a ninth of the range
// (the wider steps above would leave it a few large values, and the rest to
// round to zero).
static void fs_limbs(std::vector<double>& r, const int* pos, int nl, uint8_t* code, size_t stride, double* scale) {
  const int n = (int)r.size(), n16 = (n + 15) / 16 * 16;
  std::vector<float> rf((size_t)n16, 0.0f);  // zeros past the end leave nothing
  for (int l = 0; l < nl; ++l, code += stride) {
    for (int i = 0; i < n; ++i) rf[i] = (float)r[i];
    double mx = 0;
    for (double v : r) mx = std::max(mx, std::fabs(v));
    scale[l] = 0.0;
    if (!(mx > 0)) continue;
    const bool nearest = l + 2 >= nl;
    double best = mx / 4.5;
    if (nearest) {
      double best_err = HUGE_VAL;
      for (double f : {1.0, 0.8, 0.6}) {
        const float up = (float)(6.0 / (f * mx));
        const double s = 1.0 / (double)up;
        float err[16] = {};
        for (int i = 0; i + 16 <= n16; i += 16)
          for (int t = 0; t < 16; ++t) {
            const float v = rf[i + t] * up, d = v - e2m1_round(v);
            err[t] += d * d;
          }
        double e = 0;
        for (int t = 0; t < 16; ++t) e += err[t];
        e *= s * s;
        if (e < best_err) best_err = e, best = s;
      }
    }
    const float up = (float)(1.0 / best);
    for (int i = 0; i < n16; ++i) {
      const float t = rf[i] * up;
      rf[i] = nearest ? e2m1_round(t) : std::max(-4.0f, std::min(4.0f, near_int(t)));
    }
    for (int i = 0; i < n; ++i) {
      code[pos ? pos[i] : i] = e2m1_code(rf[i]);
      r[i] -= best * (double)rf[i];
    }
    scale[l] = best;
    if (l + 1 == nl) fs_balance(r, pos, code, best);
  }
}

static double sum_of(const std::vector<double>& r) {
  double s = 0;
  for (double v : r) s += v;
  return s;
}
static double dot(const double* a, const double* b, int n) {
  double s[4] = {0, 0, 0, 0};
  int i = 0;
  for (; i + 4 <= n; i += 4)
    for (int t = 0; t < 4; ++t) s[t] += a[i + t] * b[i + t];
  for (; i < n; ++i) s[0] += a[i] * b[i];
  return s[0] + s[1] + s[2] + s[3];
}

void column_norms(const Prepared& p, double* norm) {
  for (int j = 0; j <= p.k; ++j) {
    const double* d = &p.d[(size_t)j * p.n];
    norm[j] = std::sqrt(dot(d, d, p.n));
  }
}

void limb_loss(const Prepared& p, const double* scale, LimbLoss& B) {
  B = LimbLoss();
  column_norms(p, B.norm);
  double n2 = 0, m2 = 0;
  for (int j = 0; j <= p.k; ++j) {
    if (!(scale[j] > 0)) continue;
    const double* d = &p.d[(size_t)j * p.n];
    const double sc = scale[j], up = 1.0 / sc;  // powers of two
    double sq = 0, sum = 0;
    for (int i = 0; i < p.n; ++i) {
      const double t = d[i] * up;  // to the nearest integer, in make_limbs' way and inline
      const double r = sc * (t - (double)(long long)(t + std::copysign(0.5, t)));
      sq += r * r;
      sum += r;
    }
    if (j == p.k) {
      B.y = std::sqrt(sq) + std::fabs(sum);
    } else {
      n2 += sq;
      m2 += sum * sum;
    }
  }
  B.u = std::sqrt(n2) + std::sqrt(m2);
}

void make_fs_cols(const Prepared& p, const int* pos, int n_row, int lu, bool gate, FsCols& F) {
  const int n = p.n, k = p.k, ku = k > 0 ? k - 1 : 0;
  F = FsCols();
  F.kpad = (n_row + 255) / 256 * 256;
  F.ncol = 1 + 3 + (gate ? 4 : 0) + lu * ku;
  F.code.assign((size_t)F.ncol * F.kpad, 0);
  auto col = [&](int c) { return F.code.data() + (size_t)c * F.kpad; };
  for (int i = 0; i < n; ++i) col(0)[pos ? pos[i] : i] = e2m1_code(1.0f);
  const double* dy = &p.d[(size_t)k * n];
  std::vector<double> r(dy, dy + n);
  fs_limbs(r, pos, 3, col(1), F.kpad, F.sy);
  F.ny = std::sqrt(dot(r.data(), r.data(), n));
  F.my = std::fabs(sum_of(r)) / n;
  if (gate) {
    for (int i = 0; i < n; ++i) r[i] = dy[i];
    for (int j = 0; j < k; ++j)
      for (int i = 0; i < n; ++i) r[i] += p.g[j] * p.d[(size_t)j * n + i];
    fs_limbs(r, pos, 4, col(4), F.kpad, F.sg);
    F.ng = std::sqrt(dot(r.data(), r.data(), n));
    F.mg = std::fabs(sum_of(r)) / n;
  }
  F.su.assign((size_t)lu * ku, 0.0);
  std::vector<double> R((size_t)ku * n);
  double m2 = 0;
  for (int j = 0; j < ku; ++j) {
    const double* d = &p.d[(size_t)(j + 1) * n];
    r.assign(d, d + n);
    fs_limbs(r, pos, lu, col(4 + (gate ? 4 : 0) + lu * j), F.kpad, &F.su[(size_t)lu * j]);
    std::copy(r.begin(), r.end(), R.begin() + (size_t)j * n);
    const double s = sum_of(r) / n;
    m2 += s * s;
  }
  F.mu = std::sqrt(m2);
  // largest singular value of R: trace(G^32)^(1/32) with G = R'R / trace(R'R),
  // never below it and at most ku^(1/64) above
  std::vector<double> G((size_t)ku * ku), H((size_t)ku * ku);
  double tr = 0;
  for (int a = 0; a < ku; ++a) {
    for (int b = 0; b <= a; ++b) G[(size_t)a * ku + b] = G[(size_t)b * ku + a] = dot(&R[(size_t)a * n], &R[(size_t)b * n], n);
    tr += G[(size_t)a * ku + a];
  }
  if (tr > 0) {
    for (double& v : G) v /= tr;
    for (int it = 0; it < 5; ++it) {
      for (int a = 0; a < ku; ++a)
        for (int b = 0; b <= a; ++b)
          H[(size_t)a * ku + b] = H[(size_t)b * ku + a] = dot(&G[(size_t)a * ku], &G[(size_t)b * ku], ku);
      G.swap(H);
    }
    double t = 0;
    for (int a = 0; a < ku; ++a) t += G[(size_t)a * ku + a];
    F.nu = std::sqrt(tr * std::pow(t, 1.0 / 32));
  }
}

void put_fs_image(const FsCols& F, int col0, int N, uint8_t* img) {
  for (int c = 0; c < F.ncol; ++c) {
    const uint8_t* code = &F.code[(size_t)c * F.kpad];
    const int cc = col0 + c;
    uint8_t* base = img + (size_t)(cc >> 3) * 128 + (size_t)(cc & 7) * 16;
    for (int u = 0; u < F.kpad / 256; ++u)
      for (int cl = 0; cl < 4; ++cl)
        for (int e = 0; e < 64; e += 2) {
          // element e of the MMA: word e / 8 of the unit, its sample 4 (e % 8) + cl
          const int kap = 256 * u + 64 * cl + e;
          const uint8_t* s = code + 256 * u + 4 * e + cl;
          base[(size_t)(kap >> 5) * (N * 16) + ((kap & 31) >> 1)] = (uint8_t)(s[0] | s[4] << 4);
        }
  }
}

}  // namespace kg
