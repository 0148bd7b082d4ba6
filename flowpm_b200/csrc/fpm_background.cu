// Background cosmology on the host, FP64: the growth ODE and the kick, drift
// and LPT prefactors of a leapfrog (flowpm/tfbackground.py:533-647,
// flowpm/tfpm.py:168-177, :284-285, :306-307), with the formulas of
// flowpm_b200/tfbackground.py.  A simulation needs three prefactors per step
// before its first launch; evaluated in Python they took about 160 us per
// step and a new cosmology's growth table 20 ms, more than the leapfrog
// itself (128^3, 40 steps: 6.4 of 11.3 ms); here 30 us for the 40 steps and
// 60 us for the table.
#include <cmath>
#include <cstdint>

#include "../../include/flowpm_b200.h"

namespace {

// {Omega_m, Omega_k, Omega_de, w0, wa}
struct Cosmo {
  double om, ok, ode, w0, wa;
  // Dark-energy density exponent, tfbackground.fde (epsilon = 1e-5).
  double fde(double a) const {
    return -3.0 * (1.0 + w0) +
           3.0 * wa * ((a - 1.0) / std::log(a - 1e-5) - 1.0);
  }
  double de(double a) const { return ode * std::pow(a, fde(a)); }
  double E2(double a) const {
    return om / (a * a * a) + ok / (a * a) + de(a);
  }
  double E(double a) const { return std::sqrt(E2(a)); }
  double dEa(double a) const {
    const double la = std::log(a - 1e-5);
    const double dfde = 3 * wa * (la - (a - 1) / (a - 1e-5)) / (la * la);
    return 0.5 * (-3 * om / (a * a * a * a) - 2 * ok / (a * a * a) +
                  dfde * de(a)) / E(a);
  }
  // dy/da of the growth system y = (D1, D1', D2, D2').
  void rhs(double a, const double* y, double* r) const {
    const double e2 = E2(a);
    const double oma = om / (a * a * a) / e2;
    const double friction = de(a) / e2 - 0.5 * oma + 2.0;
    r[0] = y[1];
    r[1] = 1.5 * oma * y[0] / (a * a) - (y[1] / a) * friction;
    r[2] = y[3];
    r[3] = 1.5 * oma * y[2] / (a * a) - (y[3] / a) * friction -
           1.5 * (oma * y[0] * y[0]) / (a * a);
  }
};

Cosmo cosmo_of(const double* c) { return Cosmo{c[0], c[1], c[2], c[3], c[4]}; }

// The growth table: columns D1, D1f, D2, D2f, F1p, F2p of n values on a grid
// regular in ln a, read by linear interpolation, constant beyond its ends.
struct Growth {
  Cosmo c;
  double x0, x1;
  int n;
  const double* t;
  double at(int col, double a) const {
    double u = (std::log(a) - x0) / (x1 - x0) * (n - 1);
    u = u < 0.0 ? 0.0 : (u > n - 1.0 ? n - 1.0 : u);
    int lo = (int)std::floor(u);
    if (!(lo >= 0)) lo = 0;
    if (lo > n - 2) lo = n - 2;
    const double* y = t + (int64_t)col * n;
    return y[lo] + (u - lo) * (y[lo + 1] - y[lo]);
  }
  double D1(double a) const { return at(0, a); }
  double D1f(double a) const { return at(1, a); }
  double D2(double a) const { return at(2, a); }
  double D2f(double a) const { return at(3, a); }
  double Gf(double a) const { return D1f(a) * (a * a * a) * c.E(a); }
  // dG/da of the first (col 1, 4) or second (col 3, 5) order
  double dG(double a, int f, int fp) const {
    const double a3 = a * a * a, e = c.E(a), d = at(f, a);
    return at(fp, a) * a3 * e + d * a3 * c.dEa(a) + 3 * (a * a) * e * d;
  }
  double kick(double ai, double ac, double af) const {
    return 1 / (ac * ac * c.E(ac)) * (Gf(af) - Gf(ai)) / dG(ac, 1, 4);
  }
  double drift(double ai, double ac, double af) const {
    return 1. / (ac * ac * ac * c.E(ac)) * (D1(af) - D1(ai)) / D1f(ac);
  }
};

bool growth_of(const double* cosmo, const double* table, int n, double a0,
               double a1, Growth* g) {
  if (!cosmo || !table || n < 2 || !(a0 > 0) || !(a1 > a0)) return false;
  *g = Growth{cosmo_of(cosmo), std::log(a0), std::log(a1), n, table};
  return true;
}

}  // namespace

extern "C" int fpm_growth_ode(const double* cosmo, const double* a, int n,
                              double* y, double* dy) {
  if (!cosmo || !a || !y || !dy || n < 2) return FPM_ERR_ARG;
  const Cosmo c = cosmo_of(cosmo);
  double s[4] = {a[0], 1.0, -3.0 / 7 * (a[0] * a[0]), -6.0 / 7 * a[0]};
  for (int i = 0; i < n; ++i) {
    for (int q = 0; q < 4; ++q) y[4 * (int64_t)i + q] = s[q];
    c.rhs(a[i], s, dy + 4 * (int64_t)i);
    if (i + 1 == n) break;
    const double t = a[i], dt = a[i + 1] - a[i];
    double k[4][4], u[4];
    c.rhs(t, s, k[0]);
    for (int q = 0; q < 4; ++q) u[q] = s[q] + dt * k[0][q] / 2.0;
    c.rhs(t + dt / 2.0, u, k[1]);
    for (int q = 0; q < 4; ++q) u[q] = s[q] + dt * k[1][q] / 2.0;
    c.rhs(t + dt / 2.0, u, k[2]);
    for (int q = 0; q < 4; ++q) u[q] = s[q] + dt * k[2][q];
    c.rhs(t + dt, u, k[3]);
    for (int q = 0; q < 4; ++q)
      s[q] = s[q] + dt * (k[0][q] + 2.0 * k[1][q] + 2.0 * k[2][q] + k[3][q]) /
                        6.0;
  }
  return FPM_OK;
}

extern "C" int fpm_nbody_coefficients(const double* cosmo,
                                      const double* table, int n, double a0,
                                      double a1, const double* stages,
                                      int nstages, double* out) {
  Growth g;
  if (!growth_of(cosmo, table, n, a0, a1, &g) || nstages < 0 ||
      (nstages > 0 && !stages) || (nstages > 1 && !out))
    return FPM_ERR_ARG;
  for (int i = 0; i + 1 < nstages; ++i) {
    const double s0 = stages[i], s1 = stages[i + 1];
    const double sh = std::sqrt(s0 * s1);
    out[3 * i + 0] = g.kick(s0, s0, sh);
    out[3 * i + 1] = g.drift(s0, sh, s1);
    out[3 * i + 2] = g.kick(sh, s1, s1);
  }
  return FPM_OK;
}

extern "C" int fpm_lpt_coefficients(const double* cosmo, const double* table,
                                    int n, double a0, double a1, double a,
                                    double* out) {
  Growth g;
  if (!growth_of(cosmo, table, n, a0, a1, &g) || !out) return FPM_ERR_ARG;
  const double d1 = g.D1(a), d2 = g.D2(a), e = g.c.E(a), a2 = a * a;
  out[0] = d1;
  out[1] = d2;
  out[2] = a2 * (g.D1f(a) * a / d1) * e;
  out[3] = a2 * (g.D2f(a) * a / d2) * e;
  out[4] = a2 * e * g.dG(a, 1, 4) / d1;
  out[5] = a2 * e * g.dG(a, 3, 5) / d2;
  return FPM_OK;
}
