// Finite-difference check of the adjoint's reverses (gp_adjoint_cell.cuh) at spacings other than 1, as
// quotients and, for powers of two, as products with the reciprocals: every factor 1/dx, 1/dy, 1/(2 dy) then
// differs.  Prints <name> <max relative error> per check, compiled by tests/test_adjoint_spacing.py.
#define GP_HD inline
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "gp_adjoint_cell.cuh"

using namespace gpadj;

static double urand(double a, double b) { return a + (b - a) * (double)rand() / (double)RAND_MAX; }

template <bool POW2>
static AM<double, POW2> model(double dx, double dy, int obstacle, double fast) {
  AM<double, POW2> m = {};
  m.dx = dx; m.dy = dy; m.dt = 0.02; m.eps = 4.0; m.inv_eps = 0.25;
  m.ix = 1.0 / dx; m.iy = 1.0 / dy; m.it = 1.0 / (2.0 * dy);
  m.mob = fast / 1.7776; m.tau_ratio = 1.3; m.gam = 1.1; m.dab = 0.03;
  m.wobs = 16.0 / (M_PI * M_PI);
  m.jscale = obstacle ? -M_PI : -4.0;
  m.swell = 0.5 / sqrt(2.0);
  for (int a = 0; a < 2; a++) {
    const double th = a ? -0.4 : 0.26, c = cos(th), s = sin(th);
    m.R[a][0][0] = m.R[a][1][1] = m.Ri[a][0][0] = m.Ri[a][1][1] = c;
    m.R[a][0][1] = m.Ri[a][1][0] = -s;
    m.R[a][1][0] = m.Ri[a][0][1] = s;
  }
  m.A[0] = 1.0; m.A[1] = 0.8;
  for (int a = 0; a < 2; a++) m.cmu[a] = 1.0 / (2.0 * m.A[a]);
  m.B[0] = -0.2; m.B[1] = 0.05; m.C[0] = 0.01;
  m.Beff[0] = -0.3; m.Beff[1] = 0.15;
  m.Ds = 0.3; m.Dl = 1.2;
  m.obstacle = obstacle;
  m.skip_row = -100;
  return m;
}

// max |fd - an| over the inputs in[0 .. n), scaled by the largest difference; f: the scalar's value
template <typename F>
static double against_fd(double* in, const double* an, int n, F f) {
  double e = 0.0, scale = 1e-30;
  for (int i = 0; i < n; i++) {
    const double h = 1e-6, v = in[i];
    in[i] = v + h;
    const double up = f();
    in[i] = v - h;
    const double fd = (up - f()) / (2 * h);
    in[i] = v;
    scale = fmax(scale, fabs(fd));
    e = fmax(e, fabs(fd - an[i]));
  }
  return e / scale;
}

template <bool POW2>
static void check(const char* tag, double dx, double dy) {
  for (int kind = 0; kind < 3; kind++) {  // obstacle, well, obstacle with steps that the projection cuts
    double worst = 0.0;
    int cut = 0;
    for (int t = 0; t < 200; t++) {
      const AM<double, POW2> m = model<POW2>(dx, dy, kind != 1, kind == 2 ? 60.0 : 1.0);
      double in[19], w[2] = {urand(-1, 1), urand(-1, 1)};
      double (&P)[3][3][2] = *reinterpret_cast<double(*)[3][3][2]>(in);
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
          P[i][j][0] = kind == 2 ? urand(0.0, 1.0) : urand(0.15, 0.85);
          P[i][j][1] = 1.0 - P[i][j][0] + (kind == 2 ? 0.0 : urand(-0.02, 0.02));
        }
      if (kind == 2) P[1][1][1] = 1.0 - (P[1][1][0] = urand(0.01, 0.08));
      in[18] = urand(-0.3, 0.3);
      auto f = [&] {
        double dp[2];
        dphi_fwd(m, P, in[18], dp);
        return w[0] * dp[0] + w[1] * dp[1];
      };
      double LP[3][3][2] = {}, an[19] = {}, lpar[NPARAM] = {}, dp[2];
      dphi_fwd(m, P, in[18], dp);
      for (int a = 0; a < 2; a++) cut += P[1][1][a] + dp[a] <= 0.0 || P[1][1][a] + dp[a] >= 1.0;
      dphi_rev(m, P, in[18], w, LP, an[18], lpar);
      for (int i = 0; i < 18; i++) an[i] = (&LP[0][0][0])[i];
      worst = fmax(worst, against_fd(in, an, 19, f));
    }
    printf("%s_dphi_%s %.3e\n", tag, kind == 0 ? "obstacle" : kind == 1 ? "well" : "projected", worst);
    if (kind == 2) printf("%s_cut %d\n", tag, cut);
  }
  for (int kind = 0; kind < 3; kind++)  // diffusion flux, antitrapping current (obstacle, well); faces along x and y
    for (int dir = 0; dir < 2; dir++) {
      double worst = 0.0;
      for (int t = 0; t < 200; t++) {
        const AM<double, POW2> m = model<POW2>(dx, dy, kind != 2, 1.0);
        double in[12];
        for (int i = 0; i < 12; i++) in[i] = i < 4 ? urand(0.1, 0.9) : urand(-0.3, 0.3);
        auto face = [&] {
          Face<double> f = {{in[0], in[1]}, {in[2], in[3]}, {in[4], in[5]}, {in[6], in[7]}, in[8], in[9], in[10], in[11]};
          f.h = dir ? m.dy : m.dx;
          f.ih = dir ? m.iy : m.ix;
          f.skip = false;
          return f;
        };
        const double w = urand(-1, 1);
        FaceAdj<double> L = {};
        double lpar[NPARAM] = {};
        if (kind == 0) fface_rev(m, face(), w, L, lpar);
        else jface_rev(m, face(), w, L, lpar);
        const double an[12] = {L.pc[0], L.pc[1], L.pn[0], L.pn[1], L.tc[0], L.tc[1], L.tn[0], L.tn[1], L.muc, L.mun, L.dpc, L.dpn};
        worst = fmax(worst, against_fd(in, an, 12, [&] { return w * (kind == 0 ? fface(m, face()) : jface(m, face())); }));
      }
      printf("%s_%s_%c %.3e\n", tag, kind == 0 ? "flux" : kind == 1 ? "current_obstacle" : "current_well", dir ? 'y' : 'x', worst);
    }
  double worst = 0.0;  // the mu update of an interface cell: phi, Delta-phi, mu, the fluxes and currents
  for (int t = 0; t < 200; t++) {
    const AM<double, POW2> m = model<POW2>(dx, dy, 1, 1.0);
    double in[13];
    for (int i = 0; i < 13; i++) in[i] = i < 2 ? urand(0.1, 0.9) : i < 4 ? urand(-0.05, 0.05) : urand(-0.3, 0.3);
    const double w = urand(-1, 1);
    auto f = [&] {
      const double ph[2] = {in[0], in[1]}, dp[2] = {in[2], in[3]}, F[4] = {in[5], in[6], in[7], in[8]},
                   J[4] = {in[9], in[10], in[11], in[12]};
      return w * mu_new(m, ph, in[4], dp, F, J);
    };
    const double ph[2] = {in[0], in[1]}, dp[2] = {in[2], in[3]}, F[4] = {in[5], in[6], in[7], in[8]},
                 J[4] = {in[9], in[10], in[11], in[12]};
    double lph[2] = {0, 0}, lmu = 0, ldp[2] = {0, 0}, gdf = 0, gdj = 0;
    mu_new_rev(m, ph, in[4], dp, F, J, w, lph, lmu, ldp, gdf, gdj);
    const double an[13] = {lph[0], lph[1], ldp[0], ldp[1], lmu, gdf / dx, -gdf / dx, gdf / dy, -gdf / dy,
                           gdj * m.jscale / dx, -gdj * m.jscale / dx, gdj * m.jscale / dy, -gdj * m.jscale / dy};
    worst = fmax(worst, against_fd(in, an, 13, f));
  }
  printf("%s_mu %.3e\n", tag, worst);
}

int main() {
  srand(4321);
  check<false>("quotient", 0.7, 1.3);
  check<false>("quotient2", 0.5, 2.0);
  check<true>("product", 0.5, 2.0);
  check<true>("product4", 4.0, 0.25);
  return 0;
}
