// gp_f64.cu -- the plain form of the step: FP64, bit-faithful to the reference.
//
// Compiled with -fmad=false (and IEEE division / square root): every a*b+c
// stays a rounded multiply followed by a rounded add, as on x86-64 without
// FMA, and every expression keeps the reference's operation order, so the
// doubles produced here equal the reference solver's.
//
// Both half steps of the reference (microsim_gp.c:103-106) are pure functions of
// the pre-step state (its sweeps are Jacobi: every stencil read sees old values):
//   Delta-phi on the interior plus one ghost ring
//               (solverloop/calculate_divergence_phasefield.h:4-62);
//   antitrapping currents, mu update and phi += Delta-phi on the interior
//               (calculate_fluxes_concentration.h:4-145,
//               calculate_divergence_concentration.h:4-153), into the other
//               buffer of a double-buffered state.
// k_lean64 steps the tiles far from every interface, k_step64 the others, both half
// steps of a tile in shared memory; k_words64 makes their tile tables for a state that
// no step wrote.  k_dphi and k_update do the half steps one after the other through a
// ring array in device memory: the smoothing pre-steps, the step after a moving-frame
// shift (explicit ghost rows), models with spacings that are no powers of two or pair
// constants that are not symmetric, two-phase states most of whose tiles hold an
// interface, and the allocation-free entry.
// Ghost cells are read through gp_map (boundary copies as index maps).
//
// Reference paths are relative to Grand_potential_Finite_difference_2D_serial/.

#include <math.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "gp_common.cuh"
#include "gp_tiles.cuh"

namespace {

struct Geo {
  int mx, my;      // interior cells
  int pitch;       // elements per x-row of a state plane
  int64_t plane;   // elements per state plane
  int rpitch;      // elements per x-row of the Delta-phi ring array
  int64_t rplane;  // elements per ring plane
  gp_bc bc;
  // ghost rows y = -3..-1, my..my+2 held explicitly ([N + K1 planes][mx][6]), or
  // nullptr: ghost reads through the boundary map.  Set for the phase-field half
  // step right after a moving-frame shift, which reads the shifted ghost rows
  // before the boundary copy refreshes them (microsim_gp.c:103-125).
  const double* gov;
  // non-isothermal frozen gradient: T of ghost-padded row gy = t_bottom + gy * t_grad, for the
  // step being computed; t_linear: the phase-field half step reads the ghost rows' own linear T
  // (every step after the first: the reference resets T after the step's last boundary copy),
  // else their boundary copy
  int noniso, t_linear;
  int bc_t;  // boundary copy of T along y: 1 Neumann, 3 periodic, 0 none
  double t_bottom, t_grad;
};


// T of interior/ghost row y (interior coordinates) in the phase-field half step (linear ghosts, or
// their boundary copy in the first step) or the concentration half step (boundary copy).
__device__ __forceinline__ Th th_row(const gp_model& m, const Geo& g, int y, bool linear) {
  Th t;
  t.on = g.noniso;
  if (!g.noniso) {
    t.T = m.T;
    return t;
  }
  const int yy = (linear || !g.bc_t || (y >= 0 && y < g.my)) ? y : gp_map(y, g.my, g.bc_t);
  t.T = g.t_bottom + (double)(yy + 3) * g.t_grad;
  return t;
}

__device__ __forceinline__ const double* ghost_row(const Geo& g, int x, int y, int xtype, int q) {
  const int slot = y < 0 ? y + 3 : y - g.my + 3;
  return g.gov + ((int64_t)q * g.mx + gp_map(x, g.mx, xtype)) * 6 + slot;
}

template <int N>
__device__ __forceinline__ void load_phi(const double* __restrict__ phi, const Geo& g, int x, int y, double* out) {
  if (g.gov && (y < 0 || y >= g.my)) {
#pragma unroll
    for (int a = 0; a < N; a++) out[a] = *ghost_row(g, x, y, g.bc.phi_x, a);
    return;
  }
  const int ix = gp_map(x, g.mx, g.bc.phi_x), iy = gp_map(y, g.my, g.bc.phi_y);
  const double* p = phi + (int64_t)ix * g.pitch + iy;
#pragma unroll
  for (int a = 0; a < N; a++) out[a] = __ldg(p + a * g.plane);
}

// STABLE: no kernel that may still be running writes mu (__ldg; gp_common.cuh, dependent launches)
template <int K1, bool STABLE = true>
__device__ __forceinline__ void load_mu(const double* mu, const Geo& g, int x, int y, double* out, int nphase = 0) {
  if (g.gov && (y < 0 || y >= g.my)) {
#pragma unroll
    for (int k = 0; k < K1; k++) out[k] = *ghost_row(g, x, y, g.bc.mu_x, nphase + k);
    return;
  }
  const int ix = gp_map(x, g.mx, g.bc.mu_x), iy = gp_map(y, g.my, g.bc.mu_y);
  const double* p = mu + (int64_t)ix * g.pitch + iy;
#pragma unroll
  for (int k = 0; k < K1; k++) out[k] = STABLE ? __ldg(p + k * g.plane) : p[k * g.plane];
}

// The 3x3 phi block around (x, y).  A cell whose block lies inside the grid reads it with plain
// offsets; the others map each neighbour through the boundary copy (the same values).
template <int N>
__device__ __forceinline__ void load_block(const double* __restrict__ phi, const Geo& g, int x, int y,
                                           double (&P)[3][3][N]) {
  if (x >= 1 && x <= g.mx - 2 && y >= 1 && y <= g.my - 2) {
    const double* p = phi + (int64_t)(x - 1) * g.pitch + (y - 1);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int a = 0; a < N; a++) P[i][j][a] = __ldg(p + i * g.pitch + j + a * g.plane);
    return;
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) load_phi<N>(phi, g, x + i - 1, y + j - 1, P[i][j]);
}

// ---------------------------------------------------------------- model terms

// h_a(phi), functions/functionH.h:24-36
template <int N>
__device__ __forceinline__ double hphi(const double* phi, int a) {
  double sum1 = 0.0;
  double sum = 3.0 * phi[a] * phi[a] - 2.0 * phi[a] * phi[a] * phi[a];
#pragma unroll
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int c = b + 1; c < N; c++)
      if (b != a && c != a) sum1 += phi[b] * phi[c];
  sum1 *= 2.0 * phi[a];
  return sum + sum1;
}

// dh_b/dphi_a, functions/functionH.h:1-23 (pa, pb: phi_a, phi_b)
template <int N>
__device__ __forceinline__ double dhphi(const double* phi, double pb, double pa, int b, int a) {
  double sum = 0.0;
  if (a == b) {
    sum = 6.0 * pa * (1.0 - pa);
#pragma unroll
    for (int e = 0; e < N; e++)
#pragma unroll
      for (int f = e + 1; f < N; f++)
        if (e != b && f != b) sum += 2.0 * phi[e] * phi[f];
  } else {
#pragma unroll
    for (int e = 0; e < N; e++)
      if (e != b && e != a) sum += 2.0 * phi[e];
    sum *= pb;
  }
  return sum;
}
template <int N>
__device__ __forceinline__ double dhphi(const double* phi, int b, int a) {
  return dhphi<N>(phi, phi[b], phi[a], b, a);
}

// c_a,i(mu, T), functions/functionF_01.h:30-37
template <int K1>
__device__ __forceinline__ double c_mu(const gp_model& m, Th t, const double* mu, int a, int i) {
  double sum = 0.0;
#pragma unroll
  for (int k = 0; k < K1; k++) sum += m.cmu[a][i][k] * (mu[k] - beff(m, t, a, k));
  return sum;
}

// functions/functionF_01.h:19-29
template <int K1>
__device__ __forceinline__ double Mu(const gp_model& m, Th t, const double* c, int a, int i) {
  double sum = 2.0 * m.A[a][i][i] * c[i] + beff(m, t, a, i);
#pragma unroll
  for (int j = 0; j < K1; j++)
    if (i != j) sum += m.A[a][i][j] * c[j];
  return sum;
}

// functions/functionF_01.h:5-18, with B and C at the cell's T (init_propertymatrices(T))
template <int N, int K1>
__device__ __forceinline__ double free_energy(const gp_model& m, Th t, const double* c, int a) {
  double sum = 0.0;
#pragma unroll
  for (int i = 0; i < K1; i++) {
#pragma unroll
    for (int j = i; j < K1; j++) sum += m.A[a][i][j] * c[i] * c[j];
    sum += B_Tn<N, K1>(m, t, i, a) * c[i];
  }
  sum += C_Tn<N, K1>(m, t, a);
  return sum;
}

// d psi / d phi_a, functions/functionF_01.h:41-57
// x / d with IEEE rounding.  When d is an exact power of two the quotient equals
// the product with the exact reciprocal (one rounding of the same real number),
// so that case multiplies: the bits are those of the division, without the
// division routine (dx = dy = 1 and 2 dy = 2 in most inputs).
__device__ __forceinline__ double gp_ddiv(double x, double d) {
  const long long bits = __double_as_longlong(d);
  const long long ex = (bits >> 52) & 0x7FF;
  if ((bits & 0x000FFFFFFFFFFFFFLL) == 0 && ex > 1 && ex < 2046 && bits > 0)
    return x * __longlong_as_double((2046LL << 52) - bits);
  return x / d;
}

// a / b (IEEE, the bits of the division) from y = 1.0 / b: two residual corrections of a * y with fused
// multiply-adds, the last of which rounds correctly (P. Markstein, IBM J. Res. Develop. 34(1), 1990:
// with y the correctly rounded reciprocal and q within one unit in the last place, q + y (a - b q)
// rounds to the quotient).  Several quotients by one b then cost one division, without a branch each;
// operands near the ends of the exponent range, where a residual could leave it, and zeros divide.
__device__ __forceinline__ double quot(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  const double ma = fabs(a), mb = fabs(b);
  if (ma > 1.0e-200 && ma < 1.0e100 && mb > 1.0e-100 && mb < 1.0e100) return q;
  return a == 0.0 && b > 0.0 && mb < 1.0e300 ? a : a / b;
}

template <int N, int K1>
__device__ __forceinline__ double dpsi(const gp_model& m, Th t, const double* mu, const double* phi, int a) {
  double sum = 0.0;
#pragma unroll
  for (int b = 0; b < N; b++) {
    double c[K1];
    double psi = 0.0;
#pragma unroll
    for (int k = 0; k < K1; k++) {
      c[k] = c_mu<K1>(m, t, mu, b, k);
      psi -= mu[k] * c[k];
    }
    psi += free_energy<N, K1>(m, t, c, b);
    sum += psi * dhphi<N>(phi, b, a);
  }
  return sum;
}

// 2x2 block times vector, functions/matrix.h:22-33 with size 2
__device__ __forceinline__ void mul2(const double M[2][2], double v0, double v1, double& o0, double& o1) {
  double s = 0.0;
  s = s + M[0][0] * v0;
  s = s + M[0][1] * v1;
  o0 = s;
  s = 0.0;
  s = s + M[1][0] * v0;
  s = s + M[1][1] * v1;
  o1 = s;
}

// functions/anisotropy_01.h:30-48 (z component is 0 in 2D: dropping its +0.0
// terms is exact because the sums are non-negative)
__device__ __forceinline__ double aniso_ac(double dab, double q0, double q1) {
  const double qx2 = q0 * q0, qx4 = qx2 * qx2;
  const double qy2 = q1 * q1, qy4 = qy2 * qy2;
  const double q2 = qx2 + qy2;
  if (fabs(q2) > 1.0e-15) return 1.0 - dab * (3.0 - 4.0 * (qx4 + qy4) / (q2 * q2));
  return 1.0;
}

// functions/anisotropy_01.h:9-28
__device__ __forceinline__ void aniso_dadq(double dab, double q0, double q1, double& d0, double& d1) {
  const double qx3 = q0 * q0 * q0;
  const double qy3 = q1 * q1 * q1;
  const double q2 = q0 * q0 + q1 * q1;
  const double q22 = q2 * q2;
  const double q23 = q2 * q2 * q2;
  const double q4 = qx3 * q0 + qy3 * q1;
  if (fabs(q2) > 1.0e-15) {
    d0 = 16.0 * dab * (qx3 / q22 - q0 * q4 / q23);
    d1 = 16.0 * dab * (qy3 / q22 - q1 * q4 / q23);
  } else {
    d0 = 0.0;
    d1 = 0.0;
  }
}

// aniso_ac and aniso_dadq of one q: five quotients by |q|^4 and |q|^6
__device__ __forceinline__ void aniso_both(double dab, double q0, double q1, double& ac, double& d0, double& d1) {
  const double qx2 = q0 * q0, qx4 = qx2 * qx2;
  const double qy2 = q1 * q1, qy4 = qy2 * qy2;
  const double q2 = qx2 + qy2;
  ac = 1.0;
  d0 = d1 = 0.0;
  if (fabs(q2) > 1.0e-15) {
    const double qx3 = q0 * q0 * q0;
    const double qy3 = q1 * q1 * q1;
    const double q22 = q2 * q2;
    const double q23 = q2 * q2 * q2;
    const double q4 = qx3 * q0 + qy3 * q1;
    const double y2 = 1.0 / q22, y3 = 1.0 / q23;
    ac = 1.0 - dab * (3.0 - quot(4.0 * (qx4 + qy4), q22, y2));
    d0 = 16.0 * dab * (quot(qx3, q22, y2) - quot(q0 * q4, q23, y3));
    d1 = 16.0 * dab * (quot(qy3, q22, y2) - quot(q1 * q4, q23, y3));
  }
}

// Gradient record fields around one Delta-phi cell (calculate_gradients.h:92-131):
// the centre's full record and the parts of the four neighbours' records that
// the phase-field terms read.
template <int N>
struct Grads {
  double gx[N], gy[N], sx[N], sy[N], cx[N], cy[N];  // centre (x, y)
  double b_gx[N], b_sx[N], b_cy[N];                   // back   (x-1, y)
  double f_cy[N];                                     // front  (x+1, y)
  double l_gy[N], l_sy[N], l_cx[N];                   // left   (x, y-1)
  double r_cx[N];                                     // right  (x, y+1)
};

// P[i][j][a] = phi_a at (x+i-1, y+j-1)
template <int N>
__device__ __forceinline__ void make_grads(const gp_model& m, const double (&P)[3][3][N], double two_dy, Grads<N>& G) {
#pragma unroll
  for (int a = 0; a < N; a++) {
    G.gx[a] = gp_ddiv((P[2][1][a] - P[1][1][a]), m.dx);
    G.sx[a] = 0.5 * (P[2][1][a] + P[1][1][a]);
    G.gy[a] = gp_ddiv((P[1][2][a] - P[1][1][a]), m.dy);
    G.sy[a] = 0.5 * (P[1][2][a] + P[1][1][a]);
    G.cy[a] = gp_ddiv((P[1][2][a] - P[1][0][a]), two_dy);
    G.b_gx[a] = gp_ddiv((P[1][1][a] - P[0][1][a]), m.dx);
    G.cx[a] = 0.5 * (G.gx[a] + G.b_gx[a]);
    G.b_sx[a] = 0.5 * (P[1][1][a] + P[0][1][a]);
    G.b_cy[a] = gp_ddiv((P[0][2][a] - P[0][0][a]), two_dy);
    G.f_cy[a] = gp_ddiv((P[2][2][a] - P[2][0][a]), two_dy);
    G.l_gy[a] = gp_ddiv((P[1][1][a] - P[1][0][a]), m.dy);
    G.l_sy[a] = 0.5 * (P[1][1][a] + P[1][0][a]);
    G.l_cx[a] = 0.5 * (gp_ddiv((P[2][0][a] - P[1][0][a]), m.dx) + gp_ddiv((P[1][0][a] - P[0][0][a]), m.dx));
    G.r_cx[a] = 0.5 * (gp_ddiv((P[2][2][a] - P[1][2][a]), m.dx) + gp_ddiv((P[1][2][a] - P[0][2][a]), m.dx));
  }
}

// dA/dphi_a and div(dA/dgrad phi_a)
//   isotropic:   functions/function_A_00.h:4-58
//   anisotropic: functions/function_A_01.h:4-71, 101-219 with functionQ.h:4-72
template <int N>
__device__ __forceinline__ double grad_energy_term(const gp_model& m, const double* phi, const Grads<N>& G, int a,
                                                   bool iso = false) {
  if (!m.anisotropy || iso) {
    double sum = 0.0;
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (b == a) continue;
      double sp = 0.0;
      sp += (phi[a] * G.cx[b] - phi[b] * G.cx[a]) * G.cx[b];
      sp += (phi[a] * G.cy[b] - phi[b] * G.cy[a]) * G.cy[b];
      sp *= m.Gamma[a][b];
      sum += sp;
    }
    const double dA = 2.0 * sum;
    sum = 0.0;
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (b == a) continue;
      double dv;
      dv = gp_ddiv(((G.sx[a] * G.gx[b] - G.sx[b] * G.gx[a]) * (-G.sx[b]) -
            ((G.b_sx[a] * G.b_gx[b] - G.b_sx[b] * G.b_gx[a]) * (-G.b_sx[b]))), m.dx);
      dv += gp_ddiv(((G.sy[a] * G.gy[b] - G.sy[b] * G.gy[a]) * (-G.sy[b]) -
             ((G.l_sy[a] * G.l_gy[b] - G.l_sy[b] * G.l_gy[a]) * (-G.l_sy[b]))), m.dy);
      dv *= m.Gamma[a][b];
      sum += dv;
    }
    const double divA = 2.0 * sum;
    return -dA + divA;
  }
  // anisotropic
  double s1 = 0.0, s2 = 0.0;
#pragma unroll
  for (int b = 0; b < N; b++) {
    if (b == a) continue;
    const double gam = m.Gamma[a][b], dab = m.dab[a][b];
    double q0, q1, d0, d1, r0, r1;
    mul2(m.R[a][b], (phi[a] * G.cx[b] - phi[b] * G.cx[a]), (phi[a] * G.cy[b] - phi[b] * G.cy[a]), q0, q1);
    aniso_dadq(dab, q0, q1, d0, d1);
    const double q2 = (q0 * q0 + q1 * q1);
    const double ac1 = aniso_ac(dab, q0, q1);
    const double ac2 = ac1 * ac1;
    mul2(m.R[a][b], G.cx[b], G.cy[b], r0, r1);
    double sp1 = 0.0, sp2 = 0.0;
    sp1 += q0 * r0;
    sp1 += q1 * r1;
    sp2 += (d0)*r0;
    sp2 += (d1)*r1;
    sp1 *= gam * ac2;
    sp2 *= gam * ac1 * q2;
    s1 += sp1;
    s2 += sp2;
  }
  const double dA = 2.0 * (s1 + s2);
  s1 = 0.0;
  s2 = 0.0;
#pragma unroll
  for (int b = 0; b < N; b++) {
    if (b == a) continue;
    const double gam = m.Gamma[a][b], dab = m.dab[a][b];
    double qf0, qf1, qb0, qb1, qr0, qr1, ql0, ql1;
    mul2(m.R[a][b], (G.sx[a] * G.gx[b] - G.sx[b] * G.gx[a]),
         0.5 * (G.sx[a] * (G.cy[b] + G.f_cy[b]) - G.sx[b] * (G.cy[a] + G.f_cy[a])), qf0, qf1);
    mul2(m.R[a][b], (G.b_sx[a] * G.b_gx[b] - G.b_sx[b] * G.b_gx[a]),
         0.5 * (G.b_sx[a] * (G.b_cy[b] + G.cy[b]) - G.b_sx[b] * (G.b_cy[a] + G.cy[a])), qb0, qb1);
    mul2(m.R[a][b], 0.5 * (G.sy[a] * (G.cx[b] + G.r_cx[b]) - G.sy[b] * (G.cx[a] + G.r_cx[a])),
         (G.sy[a] * G.gy[b] - G.sy[b] * G.gy[a]), qr0, qr1);
    mul2(m.R[a][b], 0.5 * (G.l_sy[a] * (G.l_cx[b] + G.cx[b]) - G.l_sy[b] * (G.l_cx[a] + G.cx[a])),
         (G.l_sy[a] * G.l_gy[b] - G.l_sy[b] * G.l_gy[a]), ql0, ql1);
    const double acf = aniso_ac(dab, qf0, qf1), acf2 = acf * acf;
    const double acb = aniso_ac(dab, qb0, qb1), acb2 = acb * acb;
    const double acr = aniso_ac(dab, qr0, qr1), acr2 = acr * acr;
    const double acl = aniso_ac(dab, ql0, ql1), acl2 = acl * acl;
    double d1;
    d1 = gp_ddiv(((acf2 * (G.sx[a] * G.gx[b] - G.sx[b] * G.gx[a]) * (-G.sx[b])) -
          (acb2 * (G.b_sx[a] * G.b_gx[b] - G.b_sx[b] * G.b_gx[a]) * (-G.b_sx[b]))), m.dx);
    d1 += gp_ddiv(((acr2 * (G.sy[a] * G.gy[b] - G.sy[b] * G.gy[a]) * (-G.sy[b])) -
           (acl2 * (G.l_sy[a] * G.l_gy[b] - G.l_sy[b] * G.l_gy[a]) * (-G.l_sy[b]))), m.dy);
    d1 *= gam;
    s1 += d1;
    double e0, e1, rf0, rf1, rb0, rb1, rr0, rr1, rl0, rl1;
    aniso_dadq(dab, qf0, qf1, e0, e1);
    mul2(m.Rinv[a][b], e0, e1, rf0, rf1);
    const double qf2 = qf0 * qf0 + qf1 * qf1;
    aniso_dadq(dab, qb0, qb1, e0, e1);
    mul2(m.Rinv[a][b], e0, e1, rb0, rb1);
    const double qb2 = qb0 * qb0 + qb1 * qb1;
    aniso_dadq(dab, qr0, qr1, e0, e1);
    mul2(m.Rinv[a][b], e0, e1, rr0, rr1);
    const double qr2 = qr0 * qr0 + qr1 * qr1;
    aniso_dadq(dab, ql0, ql1, e0, e1);
    mul2(m.Rinv[a][b], e0, e1, rl0, rl1);
    const double ql2 = ql0 * ql0 + ql1 * ql1;
    (void)rf1; (void)rb1; (void)rr0; (void)rl0;
    double d2;
    d2 = gp_ddiv((acf * qf2 * rf0 * (-G.sx[b]) - acb * qb2 * rb0 * (-G.b_sx[b])), m.dx);
    d2 += gp_ddiv((acr * qr2 * rr1 * (-G.sy[b]) - acl * ql2 * rl1 * (-G.l_sy[b])), m.dy);
    d2 *= gam;
    s2 += d2;
  }
  const double divA = (2.0 * (s1 + s2) + 0.0);
  return -dA + divA;
}

// dw/dphi_a (pa = phi_a): obstacle functions/functionW_01.h:6-39, well functionW_02.h:4-33
template <int N>
__device__ __forceinline__ double dwdphi(const gp_model& m, const double* phi, const double* divphi, double pa, int a) {
  double sum = 0.0;
  if (m.obstacle) {
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (b == a || !(fabs(divphi[b]) > 0.0)) continue;
      if ((pa * phi[b]) >= 0.00000) sum += m.Gamma[a][b] * (phi[b]);
      else sum += -m.Gamma[a][b] * (phi[b]);
    }
    sum *= m.w_obstacle;
  } else {
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (b == a || !(fabs(divphi[b]) > 0.0)) continue;
      sum += 2.0 * m.Gamma[a][b] * (phi[b] * phi[b] * pa);
    }
    sum *= 9.0;
  }
#pragma unroll
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int c = b + 1; c < N; c++) {
      if (b == a || c == a) continue;
      if (fabs(divphi[b]) > 0.0 && fabs(divphi[c]) > 0.0) {
        const double pbc = phi[b] * phi[c];
        if (pa * pbc >= 0.00000) sum += m.Gamma_abc[a][b][c] * pbc;
        else sum += -m.Gamma_abc[a][b][c] * pbc;
      }
    }
  return sum;
}
template <int N>
__device__ __forceinline__ double dwdphi(const gp_model& m, const double* phi, const double* divphi, int a) {
  return dwdphi<N>(m, phi, divphi, phi[a], a);
}

// dw/dphi of the smoothing pre-steps with anisotropy: functionW_01.h:41-62,
// functionW_02.h:35-59 (no sign factors)
template <int N>
__device__ __forceinline__ double dwdphi_smooth(const gp_model& m, const double* phi, const double* divphi, int a) {
  double sum = 0.0;
  if (m.obstacle) {
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (b == a || !(fabs(divphi[b]) > 0.0)) continue;
      sum += m.Gamma[a][b] * phi[b];
    }
    sum *= m.w_obstacle;
  } else {
#pragma unroll
    for (int b = 0; b < N; b++) {
      if (b == a || !(fabs(divphi[b]) > 0.0)) continue;
      sum += 2.0 * m.Gamma[a][b] * (phi[b] * phi[b] * phi[a]);
    }
    sum *= 9.0;
  }
#pragma unroll
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int c = b + 1; c < N; c++) {
      if (b == a || c == a) continue;
      if (fabs(divphi[b]) > 0.0 && fabs(divphi[c]) > 0.0) sum += m.Gamma_abc[a][b][c] * phi[b] * phi[c];
    }
  return sum;
}

// functions/functionTau.h:1-16
template <int N>
__device__ __forceinline__ double tau_phi(const gp_model& m, const double* phi) {
  double sum = 0.0, sum1 = 0.0;
#pragma unroll
  for (int a = 0; a < N; a++)
#pragma unroll
    for (int b = a + 1; b < N; b++) {
      sum += m.tau_ab[a][b] * phi[a] * phi[b];
      sum1 += phi[a] * phi[b];
    }
  if (sum1 != 0.0 || sum1 != sum1) return sum / sum1;
  return m.tau;
}

// solverloop/simplex_projection.h:1-49
template <int N>
__device__ __forceinline__ void project_simplex(const double* phi, const double* divphi, double* dp) {
  double Deltaphi = 0.0, sum_phib = 0.0;
  long count = 0;
#pragma unroll
  for (int a = 0; a < N; a++)
    if ((fabs(divphi[a]) > 0.0) && (phi[a] + dp[a]) > 0.0 && (phi[a] + dp[a]) < 1.0) {
      count++;
      sum_phib += phi[a];
    }
#pragma unroll
  for (int a = 0; a < N; a++)
    if ((phi[a] + dp[a]) < 0.0) {
      const double over = fabs(dp[a] + phi[a]);
      dp[a] += over;
      Deltaphi += over;
    }
  if (Deltaphi > 0.0) {
#pragma unroll
    for (int b = 0; b < N; b++)
      if ((fabs(divphi[b]) > 0.0) && ((phi[b] + dp[b]) > 0.0) && ((phi[b] + dp[b]) < 1.0)) {
        if (fabs(sum_phib) > 0.0) dp[b] -= Deltaphi * (phi[b]) / (sum_phib);
        else dp[b] -= gp_ddiv(Deltaphi, (double)(count));
      }
  }
  int hit = -1;
#pragma unroll
  for (int a = 0; a < N; a++)
    if (hit < 0 && fabs(divphi[a]) > 0.0 && (phi[a] + dp[a]) > 1.0) hit = a;
  if (hit >= 0) {
#pragma unroll
    for (int a = 0; a < N; a++)
      if (a == hit) dp[a] = (1.0 - phi[a]);
#pragma unroll
    for (int b = 0; b < N; b++)
      if ((fabs(divphi[b]) > 0.0) && b != hit) dp[b] = -phi[b];
  }
}

// projection of the smoothing pre-steps, solverloop/simplex_projection.h:50-91
template <int N>
__device__ __forceinline__ void project_simplex_unweighted(const double* phi, const double* divphi, double* dp) {
  long count = 0;
#pragma unroll
  for (int a = 0; a < N; a++)
    if ((fabs(divphi[a]) > 0.0) && (phi[a] + dp[a]) > 0.0 && (phi[a] + dp[a]) < 1.0) count++;
  for (int a = 0; a < N; a++) {
    if (!(fabs(divphi[a]) > 0.0)) continue;
    if ((phi[a] + dp[a]) > 1.0) {
      dp[a] = (1.0 - phi[a]);
#pragma unroll
      for (int b = 0; b < N; b++)
        if ((fabs(divphi[b]) > 0.0) && b != a) dp[b] = -phi[b];
      break;
    }
    if ((phi[a] + dp[a]) < 0.0) {
      const double D = fabs(dp[a] + phi[a]);
      dp[a] += D;
#pragma unroll
      for (int b = 0; b < N; b++)
        if (((fabs(divphi[b]) > 0.0) && b != a) && (phi[b] + dp[b]) > 0.0 && (phi[b] + dp[b]) < 1.0)
          dp[b] -= gp_ddiv(D, (double)(count));
    }
  }
}

// True when the 3x3 phi block around a cell holds one value per phase and that value lies in
// [0, 1] (so no NaN, infinity or negative value).  Every phi gradient of such a cell is then
// +0 or -0: no phase is active (|divphi| = 0), the projection changes nothing, Delta-phi is
// +0, and no face next to the cell carries an antitrapping current (each face's |grad phi| is
// 0).  The kernels skip that arithmetic for such cells and store what it would give.
template <int N>
__device__ __forceinline__ bool flat_block(const double (&P)[3][3][N]) {
  bool flat = true;
#pragma unroll
  for (int a = 0; a < N; a++) {
    const double c = P[1][1][a];
    flat = flat && c >= 0.0 && c <= 1.0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) flat = flat && P[i][j][a] == c;
  }
  return flat;
}

// ---------------------------------------------------------------- kernels

// Blocks of 256 per SM the kernels are compiled for: three for binary alloys (80 registers; the
// compiler spills some of the interface cells' state, and the occupancy gained pays for it on many
// small grids stepped at once, with no loss on one large grid), two for the other two-phase
// kernels, one beyond (two of those spill heavily).
#define GP_F64_BLOCKS(N, K1) ((N) == 2 && (K1) == 1 ? 3 : ((N) == 2 ? 2 : 1))

// Delta-phi on [-1, mx] x [-1, my] (interior plus the first ghost ring).
// SMOOTH: the smoothing pre-step (calculate_divergence_phasefield.h:63-158):
// isotropic gradient energy, no dpsi, the unsigned potential when anisotropic,
// unweighted projection.
template <int N, int K1, bool SMOOTH>
__global__ void __launch_bounds__(256, GP_F64_BLOCKS(N, K1)) k_dphi(const __grid_constant__ gp_model m, Geo g,
                                              const double* __restrict__ phi, const double* __restrict__ mu,
                                              double* __restrict__ dphi) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x - 1;
  const int x = blockIdx.y * blockDim.y + threadIdx.y - 1;
  if (x > g.mx || y > g.my) return;
  double P[3][3][N];
  load_block<N>(phi, g, x, y, P);
  double* out = dphi + (int64_t)(x + 1) * g.rpitch + (y + 1);
  if (flat_block<N>(P)) {  // no active phase: Delta-phi is +0
#pragma unroll
    for (int a = 0; a < N; a++) out[a * g.rplane] = 0.0;
    return;
  }
  double muc[K1];
  load_mu<K1>(mu, g, x, y, muc, N);
  const double two_dy = 2.0 * m.dy;
  Grads<N> G;
  make_grads<N>(m, P, two_dy, G);
  const double* ph = P[1][1];
  double divphi[N], lambda[N], dp[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    divphi[a] = gp_ddiv((G.gx[a] - G.b_gx[a]), m.dx);
    divphi[a] += gp_ddiv((G.gy[a] - G.l_gy[a]), m.dy);
  }
  double sum_lambda = 0.0;
  long active = 0;
#pragma unroll
  for (int a = 0; a < N; a++) {
    lambda[a] = 0.0;
    if (fabs(divphi[a]) > 0.0) {
      const double t = grad_energy_term<N>(m, ph, G, a, SMOOTH);
      if (SMOOTH)
        lambda[a] = m.epsilon * (t) - m.inv_eps * (m.anisotropy ? dwdphi_smooth<N>(m, ph, divphi, a)
                                                                : dwdphi<N>(m, ph, divphi, a));
      else
        lambda[a] = m.epsilon * (t) - m.inv_eps * dwdphi<N>(m, ph, divphi, a) -
                    dpsi<N, K1>(m, th_row(m, g, y, g.t_linear), muc, ph, a);
      sum_lambda += lambda[a];
      active++;
    }
  }
  if (active) sum_lambda = gp_ddiv(sum_lambda, (double)active);
  const double tphi = tau_phi<N>(m, ph);
#pragma unroll
  for (int a = 0; a < N; a++) {
    if (fabs(divphi[a]) > 0.0) dp[a] = m.dt * (lambda[a] - sum_lambda) / (tphi * m.epsilon);
    else dp[a] = 0.0;
  }
  if (SMOOTH) project_simplex_unweighted<N>(ph, divphi, dp);
  else project_simplex<N>(ph, divphi, dp);
#pragma unroll
  for (int a = 0; a < N; a++) out[a * g.rplane] = dp[a];
}

// s(phi) of the obstacle antitrapping term, calculate_fluxes_concentration.h:43-59
template <int N>
__device__ __forceinline__ double s_obstacle(const double* phi, int a) {
  if (phi[a] * (1.0 - phi[a]) > 0.0) return phi[a] * (1.0 - hphi<N>(phi, a)) / (sqrt(phi[a] * (1.0 - phi[a])));
  return 0.0;
}

// Antitrapping current through the face between cell c and its neighbour n
// (n = front for an x-face, right for a y-face), one component set:
// calculate_fluxes_concentration.h:25-141.  gn: forward difference across the
// face per phase; t_c, t_n: the tangential centred gradient of c and n.
template <int N, int K1>
__device__ __forceinline__ void jat_face(const gp_model& m, const double* gn, const double* t_c, const double* t_n,
                                         const double* ph_c, const double* ph_n, const double* mu_c,
                                         const double* mu_n, const double* dp_c, const double* dp_n, bool skip,
                                         double* j, Th th_c, Th th_n) {
  constexpr int L = N - 1;
  const double tl = 0.5 * (t_c[L] + t_n[L]);
  const double norm_l = sqrt(tl * tl + gn[L] * gn[L]);
#pragma unroll
  for (int k = 0; k < K1; k++) j[k] = 0.0;
#pragma unroll
  for (int a = 0; a < N - 1; a++) {
    const double ta = 0.5 * (t_c[a] + t_n[a]);
    const double normg = sqrt(ta * ta + gn[a] * gn[a]);
    double s_n = 0.0, s_c = 0.0;
    if (m.obstacle) {
      s_n = s_obstacle<N>(ph_n, a);
      s_c = s_obstacle<N>(ph_c, a);
    }
#pragma unroll
    for (int k = 0; k < K1; k++) {
      if (normg != 0.0 && !skip) {
        const double cl_n = c_mu<K1>(m, th_n, mu_n, L, k), cl_c = c_mu<K1>(m, th_c, mu_c, L, k);
        const double cs_n = c_mu<K1>(m, th_n, mu_n, a, k), cs_c = c_mu<K1>(m, th_c, mu_c, a, k);
        double sp = gn[a] * gn[L];
        sp += ta * tl;
        if (norm_l > 0.0) sp /= (norm_l * normg);
        const double f = (1.0 - m.Diff[a][k][k] / m.Diff[L][k][k]);
        if (m.obstacle)
          j[k] += f * fabs(sp) * 0.5 * (s_n * (cl_n - cs_n) * dp_n[a] + s_c * (cl_c - cs_c) * dp_c[a]) * gn[a] / normg;
        else
          j[k] += f * fabs(sp) * m.s_well * ((cl_n - cs_n) * dp_n[a] + (cl_c - cs_c) * dp_c[a]) * gn[a] / normg;
      }
    }
  }
}

// phi-weighted mobility of one cell, functions/functionD.h:1-16
template <int N, int K1>
__device__ __forceinline__ double Dcell(const gp_model& m, const double* phi, int i, int j) {
  double sum = 0.0;
#pragma unroll
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int k = 0; k < K1; k++) sum += m.Diff[b][i][k] * m.cmu[b][k][j] * phi[b];
  return sum;
}

// LU inverse of the reference (functions/matrix.h:50-114) for the general mu solve.
template <int K>
__device__ __forceinline__ void lu_inverse(double (&mm)[K][K], double (&inv)[K][K]) {
  double fac[K][K], inv1[K][K];
  int tag[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    tag[k] = k;
#pragma unroll
    for (int j = 0; j < K; j++) fac[k][j] = 0.0;
  }
#pragma unroll
  for (int k = 0; k < K; k++) {
    double big = fabs(mm[k][k]);
    int t1 = k;
#pragma unroll
    for (int i = k + 1; i < K; i++)
      if (fabs(mm[i][k]) > big) { t1 = i; big = mm[i][k]; }
    // swap tag[k] <-> tag[t1], rows k <-> t1 of mm, and fac[.][0..k-1]
#pragma unroll
    for (int i = k + 1; i < K; i++) {
      if (i == t1) {
        int ts = tag[k]; tag[k] = tag[i]; tag[i] = ts;
#pragma unroll
        for (int c = 0; c < K; c++) { double s = mm[k][c]; mm[k][c] = mm[i][c]; mm[i][c] = s; }
#pragma unroll
        for (int c = 0; c < k; c++) { double s = fac[k][c]; fac[k][c] = fac[i][c]; fac[i][c] = s; }
      }
    }
#pragma unroll
    for (int i = k + 1; i < K; i++) {
      const double f = -mm[i][k] / mm[k][k];
      fac[i][k] = -f;
#pragma unroll
      for (int j = k; j <= K - 1; j++) mm[i][j] = f * mm[k][j] + mm[i][j];
    }
  }
#pragma unroll
  for (int i = 0; i < K; i++)
#pragma unroll
    for (int j = 0; j < K; j++) {
      if (i == j) fac[i][j] = 1;
      if (j > i) fac[i][j] = 0;
    }
#pragma unroll
  for (int i = 0; i < K; i++) {
    double v1[K], v[K];
    v1[0] = (i == 0) ? 1.0 : 0.0;
#pragma unroll
    for (int k = 1; k < K; k++) {
      double s = 0;
#pragma unroll
      for (int j = 0; j < k; j++) s = s - fac[k][j] * v1[j];
      v1[k] = ((k == i) ? 1.0 : 0.0) + s;
    }
    // pow(x, -1) of the reference equals the correctly rounded 1/x
    v[K - 1] = v1[K - 1] * (1.0 / mm[K - 1][K - 1]);
#pragma unroll
    for (int k = K - 2; k >= 0; k--) {
      double s = 0;
#pragma unroll
      for (int j = k + 1; j < K; j++) s = s - mm[k][j] * v[j];
      v[k] = (v1[k] + s) * (1.0 / mm[k][k]);
    }
#pragma unroll
    for (int j = 0; j < K; j++) inv1[j][i] = v[j];
  }
#pragma unroll
  for (int j = 0; j < K; j++)
#pragma unroll
    for (int t = 0; t < K; t++)
      if (tag[j] == t) {
#pragma unroll
        for (int k = 0; k < K; k++) inv[k][t] = inv1[k][j];
      }
}

// Division by the grid spacings: IEEE quotients, or products with their exact reciprocals where the
// spacings are powers of two (the same bits; gp_ddiv).
struct DivSpacing {
  double hx, hy;
  __device__ __forceinline__ double dx(double v) const { return gp_ddiv(v, hx); }
  __device__ __forceinline__ double dy(double v) const { return gp_ddiv(v, hy); }
};
struct MulSpacing {
  double ix, iy;
  __device__ __forceinline__ double dx(double v) const { return v * ix; }
  __device__ __forceinline__ double dy(double v) const { return v * iy; }
};

// New mu of a cell from its own and its four neighbours' phi and mu, its Delta-phi and the currents
// of its four faces.  SMOOTH: the smoothing pre-step (no current, no dh/dt source, the LU inverse).
template <int N, int K1, bool SMOOTH, typename S>
__device__ __forceinline__ void cell_update(const gp_model& m, const S& sp, Th thc, const double* ph, const double* phb,
                                            const double* phf, const double* phl, const double* phr,
                                            const double* Mc, const double* Mb, const double* Mf, const double* Ml,
                                            const double* Mr, const double* Dc, const double* jx_c,
                                            const double* jx_b, const double* jy_c, const double* jy_l,
                                            double (&mnew)[K1]) {
  double sum[K1], divflux[K1], divjat[K1], deltac[K1], dcdmu[K1][K1];
#pragma unroll
  for (int k = 0; k < K1; k++) {
    sum[k] = 0.0;
#pragma unroll
    for (int l = 0; l < K1; l++) dcdmu[k][l] = 0.0;
  }
#pragma unroll
  for (int a = 0; a < N; a++) {
    double sdh = 0.0;
#pragma unroll
    for (int b = 0; b < N; b++) sdh += dhphi<N>(ph, a, b) * Dc[b];
#pragma unroll
    for (int k = 0; k < K1; k++) sum[k] += c_mu<K1>(m, thc, Mc, a, k) * sdh;
  }
  const double jscale = m.obstacle ? m.jat_obst : m.jat_well;
#pragma unroll
  for (int k = 0; k < K1; k++) {
    divflux[k] = 0.0;
#pragma unroll
    for (int l = 0; l < K1; l++) {
      const double Dcc = Dcell<N, K1>(m, ph, k, l);
      const double Dx = (Dcell<N, K1>(m, phf, k, l) + Dcc) * 0.5;
      const double Dxb = (Dcc + Dcell<N, K1>(m, phb, k, l)) * 0.5;
      const double Dy = (Dcell<N, K1>(m, phr, k, l) + Dcc) * 0.5;
      const double Dyl = (Dcc + Dcell<N, K1>(m, phl, k, l)) * 0.5;
      const double gmx = sp.dx((Mf[l] - Mc[l]));
      const double gmxb = sp.dx((Mc[l] - Mb[l]));
      const double gmy = sp.dy((Mr[l] - Mc[l]));
      const double gmyl = sp.dy((Mc[l] - Ml[l]));
      divflux[k] += sp.dx((Dx * gmx - Dxb * gmxb));
      divflux[k] += sp.dy((Dy * gmy - Dyl * gmyl));
    }
    if (!SMOOTH) {
      divjat[k] = sp.dx((jx_c[k] - jx_b[k]) * (jscale));
      divjat[k] += sp.dy((jy_c[k] - jy_l[k]) * (jscale));
    }
  }
  int bulk = -1;
#pragma unroll
  for (int a = 0; a < N; a++)
    if (bulk < 0 && ph[a] == 1.0) bulk = a;
  if (bulk >= 0) {
    double cnew[K1];
#pragma unroll
    for (int k = 0; k < K1; k++) {
      double co = 0.0;
#pragma unroll
      for (int a = 0; a < N; a++)
        if (a == bulk) co = c_mu<K1>(m, thc, Mc, a, k);
      cnew[k] = SMOOTH ? co + m.dt * (divflux[k]) : co + m.dt * (divflux[k]) - divjat[k];
    }
#pragma unroll
    for (int k = 0; k < K1; k++) {
      double v = 0.0;
#pragma unroll
      for (int a = 0; a < N; a++)
        if (a == bulk) v = Mu<K1>(m, thc, cnew, a, k);
      mnew[k] = v;
    }
  } else if (SMOOTH) {
#pragma unroll
    for (int k = 0; k < K1; k++) {
      deltac[k] = m.dt * (divflux[k]);
#pragma unroll
      for (int l = 0; l < K1; l++)
#pragma unroll
        for (int a = 0; a < N; a++) dcdmu[k][l] += m.cmu[a][k][l] * hphi<N>(ph, a);
    }
    double inv[K1][K1];
    lu_inverse<K1>(dcdmu, inv);
#pragma unroll
    for (int k = 0; k < K1; k++) {
      double s = 0;
#pragma unroll
      for (int l = 0; l < K1; l++) s = s + inv[k][l] * deltac[l];
      mnew[k] = s + Mc[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < K1; k++) {
      deltac[k] = m.dt * (divflux[k]) - divjat[k] - sum[k];
#pragma unroll
      for (int l = 0; l < K1; l++)
#pragma unroll
        for (int a = 0; a < N; a++) dcdmu[k][l] += m.cmu[a][k][l] * hphi<N>(ph, a);
    }
#pragma unroll
    for (int k = 0; k < K1; k++) mnew[k] = Mc[k];
    if (m.mu_solver == GP_MU_BINARY) {
      const double iv = 1.0 / dcdmu[0][0];
      mnew[0] = Mc[0] + deltac[0] * iv;
    } else if (m.mu_solver == GP_MU_TERNARY && K1 == 2) {
      const double DET = dcdmu[0][0] * dcdmu[K1 - 1][K1 - 1] - dcdmu[0][K1 - 1] * dcdmu[K1 - 1][0];
      double inv[2][2];
      const double yd = 1.0 / DET;
      inv[0][0] = quot(dcdmu[K1 - 1][K1 - 1], DET, yd);
      inv[1][1] = quot(dcdmu[0][0], DET, yd);
      inv[0][1] = quot(-dcdmu[0][K1 - 1], DET, yd);
      inv[1][0] = quot(-dcdmu[K1 - 1][0], DET, yd);
#pragma unroll
      for (int k = 0; k < K1; k++) {
        double dm = 0.0;
#pragma unroll
        for (int l = 0; l < K1; l++) dm += inv[k & 1][l & 1] * deltac[l];
        mnew[k] = dm + Mc[k];
      }
    } else if (m.mu_solver == GP_MU_DILUTE) {
#pragma unroll
      for (int k = 0; k < K1; k++) {
        const double iv = 1.0 / dcdmu[k][k];
        mnew[k] = Mc[k] + deltac[k] * iv;
      }
    } else {
      double inv[K1][K1];
      lu_inverse<K1>(dcdmu, inv);
#pragma unroll
      for (int k = 0; k < K1; k++) {
        double s = 0;
#pragma unroll
        for (int l = 0; l < K1; l++) s = s + inv[k][l] * deltac[l];
        mnew[k] = s + Mc[k];
      }
    }
  }
}

// mu and phi update of the interior.  SMOOTH: the smoothing pre-step
// (calculate_divergence_concentration.h:154-253): no antitrapping current, no
// dh/dt source, the LU inverse (matinvnew) for every mu solve.
template <int N, int K1, bool SMOOTH>
__global__ void __launch_bounds__(256, GP_F64_BLOCKS(N, K1)) k_update(const __grid_constant__ gp_model m, Geo g,
                                                const double* __restrict__ phi, const double* __restrict__ mu,
                                                const double* __restrict__ dphi, double* __restrict__ phi_out,
                                                double* __restrict__ mu_out) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= g.mx || y >= g.my) return;
  double P[3][3][N];
  load_block<N>(phi, g, x, y, P);
  double Mc[K1], Mb[K1], Mf[K1], Ml[K1], Mr[K1];
  if (x >= 1 && x <= g.mx - 2 && y >= 1 && y <= g.my - 2) {  // the four neighbours inside the grid
    const double* q = mu + (int64_t)x * g.pitch + y;
#pragma unroll
    for (int k = 0; k < K1; k++) {
      Mc[k] = __ldg(q + k * g.plane);
      Mb[k] = __ldg(q + k * g.plane - g.pitch);
      Mf[k] = __ldg(q + k * g.plane + g.pitch);
      Ml[k] = __ldg(q + k * g.plane - 1);
      Mr[k] = __ldg(q + k * g.plane + 1);
    }
  } else {
    load_mu<K1>(mu, g, x, y, Mc);
    load_mu<K1>(mu, g, x - 1, y, Mb);
    load_mu<K1>(mu, g, x + 1, y, Mf);
    load_mu<K1>(mu, g, x, y - 1, Ml);
    load_mu<K1>(mu, g, x, y + 1, Mr);
  }
  double Dc[N], Db[N], Df[N], Dl[N], Dr[N];
  {
    const double* r = dphi + (int64_t)(x + 1) * g.rpitch + (y + 1);
#pragma unroll
    for (int a = 0; a < N; a++) {
      Dc[a] = __ldg(r + a * g.rplane);
      Db[a] = __ldg(r + a * g.rplane - g.rpitch);
      Df[a] = __ldg(r + a * g.rplane + g.rpitch);
      Dl[a] = __ldg(r + a * g.rplane - 1);
      Dr[a] = __ldg(r + a * g.rplane + 1);
    }
  }
  // j_at on the four faces; the y-face at ghosted row MESH_Y-2 carries none
  // (calculate_fluxes_concentration.h:65), i.e. interior row my-5.  A flat phi block
  // carries none on any face (flat_block).
  double jx_c[K1], jx_b[K1], jy_c[K1], jy_l[K1];
#pragma unroll
  for (int k = 0; k < K1; k++) jx_c[k] = jx_b[k] = jy_c[k] = jy_l[k] = 0.0;
  // the cells' temperatures in the concentration half step (ghosts: their boundary copy)
  const Th thc = th_row(m, g, y, false), thl = th_row(m, g, y - 1, false), thr = th_row(m, g, y + 1, false);
  if (!SMOOTH && !flat_block<N>(P)) {
    const double two_dy = 2.0 * m.dy;
    // gradient pieces the four faces need (calculate_gradients.h:92-131)
    double gx_c[N], gx_b[N], gy_c[N], gy_l[N];
    double cy_c[N], cy_b[N], cy_f[N], cx_c[N], cx_l[N], cx_r[N];
#pragma unroll
    for (int a = 0; a < N; a++) {
      gx_c[a] = gp_ddiv((P[2][1][a] - P[1][1][a]), m.dx);
      gx_b[a] = gp_ddiv((P[1][1][a] - P[0][1][a]), m.dx);
      gy_c[a] = gp_ddiv((P[1][2][a] - P[1][1][a]), m.dy);
      gy_l[a] = gp_ddiv((P[1][1][a] - P[1][0][a]), m.dy);
      cy_c[a] = gp_ddiv((P[1][2][a] - P[1][0][a]), two_dy);
      cy_b[a] = gp_ddiv((P[0][2][a] - P[0][0][a]), two_dy);
      cy_f[a] = gp_ddiv((P[2][2][a] - P[2][0][a]), two_dy);
      cx_c[a] = 0.5 * (gx_c[a] + gx_b[a]);
      cx_l[a] = 0.5 * (gp_ddiv((P[2][0][a] - P[1][0][a]), m.dx) + gp_ddiv((P[1][0][a] - P[0][0][a]), m.dx));
      cx_r[a] = 0.5 * (gp_ddiv((P[2][2][a] - P[1][2][a]), m.dx) + gp_ddiv((P[1][2][a] - P[0][2][a]), m.dx));
    }
    jat_face<N, K1>(m, gx_c, cy_c, cy_f, P[1][1], P[2][1], Mc, Mf, Dc, Df, false, jx_c, thc, thc);
    jat_face<N, K1>(m, gx_b, cy_b, cy_c, P[0][1], P[1][1], Mb, Mc, Db, Dc, false, jx_b, thc, thc);
    jat_face<N, K1>(m, gy_c, cx_c, cx_r, P[1][1], P[1][2], Mc, Mr, Dc, Dr, (y + 3 == g.my - 2), jy_c, thc, thr);
    jat_face<N, K1>(m, gy_l, cx_l, cx_c, P[1][0], P[1][1], Ml, Mc, Dl, Dc, (y + 2 == g.my - 2) || (y + 2 == 0),
                    jy_l, thl, thc);
  }

  const double* ph = P[1][1];
  double mnew[K1];
  cell_update<N, K1, SMOOTH>(m, DivSpacing{m.dx, m.dy}, thc, ph, P[0][1], P[2][1], P[1][0], P[1][2], Mc, Mb, Mf, Ml, Mr, Dc, jx_c, jx_b, jy_c,
                             jy_l, mnew);
  const int64_t o = (int64_t)x * g.pitch + y;
#pragma unroll
  for (int k = 0; k < K1; k++) mu_out[o + k * g.plane] = mnew[k];
#pragma unroll
  for (int a = 0; a < N; a++) phi_out[o + a * g.plane] = ph[a] + Dc[a];
}

// ---------------------------------------------------------------- the tile kernel

// Constants of the tile kernel folded on the host (IEEE, the kernels' operation order).
struct C64 {
  double ix, iy, i2y;                       // exact reciprocals of dx, dy, 2 dy (powers of two)
  double atf[GP_MAX_PHASES][GP_MAX_K1];     // 1 - Diff_a / Diff_liquid
  double Dp[GP_MAX_PHASES][GP_MAX_K1][GP_MAX_K1];  // mobility of the pure phase (Dcell of its one-hot phi)
};

// A tile of 8 x 16 cells, two threads per cell.  Shared memory, in doubles.
template <int N, int K1>
struct T64 {
  static constexpr int TX = 8, TY = 16, NT = 2 * TX * TY;
  static constexpr int X1 = TX + 2, Y1 = TY + 2, X2 = TX + 4, Y2 = TY + 4;  // tile +- 1 (ring), +- 2
  static constexpr int P = N * (N - 1) / 2;
  static constexpr int FX = (TX + 3) * Y1, NF = FX + X1 * (TY + 3);   // x-, all faces of the ring's cells
  static constexpr int JX = (TX + 1) * TY, NJ = JX + TX * (TY + 1);   // x-, all faces of the tile's cells
  static constexpr int o_phi = 0;                    // [N][X2][Y2]
  static constexpr int o_mu = o_phi + N * X2 * Y2;   // [K1][X1][Y1]
  static constexpr int o_dp = o_mu + K1 * X1 * Y1;   // [N][X1][Y1] lambda, then Delta-phi
  static constexpr int o_face = o_dp + N * X1 * Y1;  // [P][2][NF] gradient-energy face terms, then
  static constexpr int n_cur = K1 * NJ + (N - 1) * X1 * Y1;  // antitrapping currents [K1][NJ], s(phi) [N-1][X1][Y1]
  static constexpr int total = o_face + (2 * P * NF > n_cur ? 2 * P * NF : n_cur);
  static constexpr size_t bytes = total * sizeof(double);
  static constexpr int unroll = N <= 4 ? N : 1;
  static constexpr int blocks = N <= 4 ? 2 : 1;  // resident blocks per SM asked of the compiler
};

// asynchronous 8-byte copy to shared memory (cp.async), complete after cp.async.wait_all
__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <int N>
__device__ __forceinline__ void pair_of(int p, int& a, int& b) {  // pairs a < b in the order (0,1), (0,2), ...
  a = 0;
  while (p >= N - 1 - a) p -= N - 1 - a++;
  b = a + 1 + p;
}
template <int N>
__device__ __forceinline__ int pair_index(int a, int b) { return a * N - a * (a + 1) / 2 + (b - a - 1); }

// Purity word of a tile (gp_tiles.cuh) from the classes (the phase a cell is the one-hot field of, 0xFF for
// none) of its corner cells (0, 0), (ex - 1, 0), (0, ey - 1) and the parts in which some cell differs.
__device__ __forceinline__ uint32_t part_bits(int TXi, int TYj, int ex, int ey, int v, int r0, int rxh, int ryh) {
  uint32_t bad = 0u;
  if (v != r0) bad |= (TXi < 2 ? 3u : 1u) | (TYj < 2 ? 8u : 0u);
  if (TXi >= ex - 2 && v != rxh) bad |= 4u;
  if (TYj >= ey - 2 && v != ryh) bad |= 16u;
  return bad;
}
__device__ __forceinline__ uint32_t word_of(uint32_t bad, int r0, int rxh, int ryh) {
  uint32_t w = 0u;
  if (!(bad & 1u) && r0 != 0xFF) w |= (uint32_t)(1 + r0) << PF_CORE;
  if (!(bad & 2u) && r0 != 0xFF) w |= (uint32_t)(1 + r0) << PF_XLO;
  if (!(bad & 4u) && rxh != 0xFF) w |= (uint32_t)(1 + rxh) << PF_XHI;
  if (!(bad & 8u) && r0 != 0xFF) w |= (uint32_t)(1 + r0) << PF_YLO;
  if (!(bad & 16u) && ryh != 0xFF) w |= (uint32_t)(1 + ryh) << PF_YHI;
  return w;
}

// New mu of a bulk cell of phase b all of whose neighbours hold the one-hot phi of b: what cell_update
// yields there (no current, face mobility (D + D) / 2).  u: centre, x-, x+, y-, y+.
template <int N, int K1>
__device__ __forceinline__ void pure_cell(const gp_model& m, const C64& c64, Th th, int b, const double (&u)[5][K1],
                                          double (&mnew)[K1]) {
  const double ix = c64.ix, iy = c64.iy, jscale = m.obstacle ? m.jat_obst : m.jat_well;
  double cnew[K1];
#pragma unroll
  for (int k = 0; k < K1; k++) {
    double divflux = 0.0;
#pragma unroll
    for (int l = 0; l < K1; l++) {
      const double D = c64.Dp[b][k][l], Dx = (D + D) * 0.5;
      const double gmx = (u[2][l] - u[0][l]) * ix, gmxb = (u[0][l] - u[1][l]) * ix;
      const double gmy = (u[4][l] - u[0][l]) * iy, gmyl = (u[0][l] - u[3][l]) * iy;
      divflux += (Dx * gmx - Dx * gmxb) * ix;
      divflux += (Dx * gmy - Dx * gmyl) * iy;
    }
    double divjat = ((0.0 - 0.0) * (jscale)) * ix;
    divjat += ((0.0 - 0.0) * (jscale)) * iy;
    cnew[k] = c_mu<K1>(m, th, u[0], b, k) + m.dt * (divflux)-divjat;
  }
#pragma unroll
  for (int k = 0; k < K1; k++) mnew[k] = Mu<K1>(m, th, cnew, b, k);
}

// Purity words of a state that no step wrote (an upload, a caller's writes, smoothing, a shift), nothing known of
// the other buffer (its words 0) and both list counts 0: a warp per tile, the lanes' cells as in k_lean64.
// One read of phi, where a step without words takes every tile through k_step64: a 1024^2 dendrite whose
// state changes every step takes 33 us per step, 86 without this and 46 through the ring array.
template <int N, int K1>
__global__ void __launch_bounds__(256) k_words64(Geo g, const double* __restrict__ phi, uint32_t* __restrict__ words,
                                                 uint32_t* __restrict__ other, int* __restrict__ cnt, int ntile) {
  constexpr int TX = T64<N, K1>::TX, TY = T64<N, K1>::TY;
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x < 2) cnt[threadIdx.x] = 0;
  if (t >= ntile) return;
  const int nty = (g.my + TY - 1) / TY, x0 = (t / nty) * TX, y0 = (t % nty) * TY;
  const int ex = min(TX, g.mx - x0), ey = min(TY, g.my - y0), i0 = lane >> 3, j0 = 2 * (lane & 7);
  double2 v[2][N];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int x = min(x0 + i0 + 4 * r, g.mx - 1);  // (a row's padding lies within its pitch)
#pragma unroll
    for (int a = 0; a < N; a++)
      v[r][a] = __ldg(reinterpret_cast<const double2*>(phi + a * g.plane + (int64_t)x * g.pitch + y0 + j0));
  }
  int cls[2][2];
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      int hot = -1;
      bool onehot = true;
#pragma unroll
      for (int a = 0; a < N; a++) {
        const double p = c ? v[r][a].y : v[r][a].x;
        if (p == 1.0 && hot < 0) hot = a;
        else if (__double_as_longlong(p) != 0) onehot = false;  // -0 is not the pure field's +0
      }
      cls[r][c] = onehot && hot >= 0 ? hot : 0xFF;
    }
  constexpr unsigned ALL = 0xffffffffu;
  const int r0 = __shfl_sync(ALL, cls[0][0], 0);
  const int xr = ex - 1, xlane = (xr & 3) * 8, h0 = __shfl_sync(ALL, cls[0][0], xlane), h1 = __shfl_sync(ALL, cls[1][0], xlane);
  const int yc = ey - 1, y_0 = __shfl_sync(ALL, cls[0][0], yc >> 1), y_1 = __shfl_sync(ALL, cls[0][1], yc >> 1);
  const int rxh = xr >= 4 ? h1 : h0, ryh = yc & 1 ? y_1 : y_0;
  uint32_t bad = 0u;
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const int i = i0 + 4 * r, j = j0 + c;
      if (i < ex && j < ey) bad |= part_bits(i, j, ex, ey, cls[r][c], r0, rxh, ryh);
    }
  bad = __reduce_or_sync(ALL, bad);
  if (lane == 0) {
    words[t] = word_of(bad, r0, rxh, ryh);
    other[t] = 0u;
  }
}

// The step of the tiles that lean_phase accepts: they hold the one-hot field of one phase on their
// cells and the two rings a step reads, so Delta-phi is +0, no face carries an antitrapping current
// and every cell is bulk: mu alone moves, and phi is written only where the output buffer does not
// hold that field yet (its purity word says so).  The other tiles are listed for k_step64.
// A warp per tile, two cells of two rows per lane (16-byte loads).  win, wout: purity words of the
// input and the output buffer (gp_tiles.cuh); cnt[0] counts the list.
// Bound by latency: tile facts, nine words and mu are a chain of three loads, and one wave of blocks
// covers a 1024^2 grid.
template <int N, int K1>
__global__ void __launch_bounds__(256) k_lean64(const __grid_constant__ gp_model m, const __grid_constant__ C64 c64,
                                                Geo g, const uint32_t* __restrict__ geo,
                                                const uint32_t* win, uint32_t* wout, int ntile, const double* mu,
                                                double* phi_out, double* mu_out, int* list, int* cnt) {
  constexpr int TX = T64<N, K1>::TX, TY = T64<N, K1>::TY;
  gp_allow_dependents();  // the list's reader
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= ntile) return;
  const uint32_t tg = geo[t];
  gp_wait_for_earlier_kernels();
  const int b = lean_phase(win, tg, t);
  if (b < 0) {
    if (lane == 0) list[atomicAdd(cnt, 1)] = t;
    return;
  }
  const bool write_phi = pf(wout[t], PF_CORE) != 1 + b;
  const int nty = (g.my + TY - 1) / TY, x0 = (t / nty) * TX, y0 = (t % nty) * TY;
  const int xr = x0 + (lane >> 3), y = y0 + 2 * (lane & 7);
  if (x0 > 0 && x0 + TX < g.mx && y0 > 0 && y0 + TY < g.my) {
    double2 u[2][3][K1];
    double ul[2][K1], ur[2][K1];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int k = 0; k < K1; k++) {
        const double* p = mu + k * g.plane + (int64_t)(xr + 4 * r) * g.pitch + y;
        u[r][0][k] = *reinterpret_cast<const double2*>(p);
        u[r][1][k] = *reinterpret_cast<const double2*>(p - g.pitch);
        u[r][2][k] = *reinterpret_cast<const double2*>(p + g.pitch);
        ul[r][k] = p[-1];
        ur[r][k] = p[2];
      }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      double c0[5][K1], c1[5][K1], m0[K1], m1[K1];
#pragma unroll
      for (int k = 0; k < K1; k++) {
        c0[0][k] = u[r][0][k].x; c0[1][k] = u[r][1][k].x; c0[2][k] = u[r][2][k].x; c0[3][k] = ul[r][k]; c0[4][k] = u[r][0][k].y;
        c1[0][k] = u[r][0][k].y; c1[1][k] = u[r][1][k].y; c1[2][k] = u[r][2][k].y; c1[3][k] = u[r][0][k].x; c1[4][k] = ur[r][k];
      }
      pure_cell<N, K1>(m, c64, th_row(m, g, y, false), b, c0, m0);
      pure_cell<N, K1>(m, c64, th_row(m, g, y + 1, false), b, c1, m1);
      const int64_t o = (int64_t)(xr + 4 * r) * g.pitch + y;
#pragma unroll
      for (int k = 0; k < K1; k++) *reinterpret_cast<double2*>(mu_out + o + k * g.plane) = make_double2(m0[k], m1[k]);
      if (write_phi) {
#pragma unroll
        for (int a = 0; a < N; a++) {
          const double v = a == b ? 1.0 : 0.0;
          *reinterpret_cast<double2*>(phi_out + o + a * g.plane) = make_double2(v, v);
        }
      }
    }
  } else {  // a tile at the grid's edge: cell by cell through the boundary map
#pragma unroll 1
    for (int q = 0; q < 4; q++) {
      const int x = xr + 4 * (q >> 1), yq = y + (q & 1);
      if (x >= g.mx || yq >= g.my) continue;
      double u[5][K1], mnew[K1];
      load_mu<K1, false>(mu, g, x, yq, u[0]);
      load_mu<K1, false>(mu, g, x - 1, yq, u[1]);
      load_mu<K1, false>(mu, g, x + 1, yq, u[2]);
      load_mu<K1, false>(mu, g, x, yq - 1, u[3]);
      load_mu<K1, false>(mu, g, x, yq + 1, u[4]);
      pure_cell<N, K1>(m, c64, th_row(m, g, yq, false), b, u, mnew);
      const int64_t o = (int64_t)x * g.pitch + yq;
#pragma unroll
      for (int k = 0; k < K1; k++) mu_out[o + k * g.plane] = mnew[k];
      if (write_phi) {
#pragma unroll
        for (int a = 0; a < N; a++) phi_out[o + a * g.plane] = a == b ? 1.0 : 0.0;
      }
    }
  }
  __syncwarp();
  if (lane == 0) wout[t] = pf_all(1 + b);
}

// The step of the listed tiles (blocks take entries blockIdx.x, + gridDim.x, ...), each through
// shared memory.
//
// What each step of the arithmetic yields is what k_dphi and k_update yield: the same expressions
// in the same order.  What is evaluated once instead of two or four times: the gradient-energy
// terms of a face (the front face of one cell is the back face of the next: the same operands in
// the same order), those of the pairs (a, b) and (b, a) (q, its anisotropy derivative and Q_n only
// change sign), s(phi) of a cell and a face's antitrapping current.  The host sends models here whose
// pair constants are symmetric and whose spacings are powers of two (division is a product).
//
// Bound by instruction fetch, then latency: a launch holds few interface tiles, each runs the
// whole chain stage -> flags -> face terms -> lambda -> Delta-phi -> currents -> update once, and
// warps wait for its code (no_instruction is the first stall reason).  So every phase is one copy of
// its code: x- and y-faces share a loop through strides, phases and pairs are items spread over the
// threads or rolled loops, and no division by a spacing is left.  Tiles of 128 cells spread an
// interface over twice the SMs of 8 x 32 ones.
// A step with k_lean64, against k_dphi and k_update: 1024^2 dendrite 43.4 -> 24.2 us, 611x500 four-phase
// ternary 242 -> 127, 300x451 frozen gradient 43 -> 28, 200^2 22 -> 18; one kernel over 8 x 32 tiles for
// bulk and interface was slower than the two it replaced (0.83x on the dendrite).
template <int N, int K1>
__global__ void __launch_bounds__(T64<N, K1>::NT, T64<N, K1>::blocks)
    k_step64(const __grid_constant__ gp_model m, const __grid_constant__ C64 c64, Geo g, uint32_t* wout,
             const double* phi, const double* mu, double* phi_out, double* mu_out, const int* list, const int* cnt,
             int* next_cnt, int* seen, int* told) {
  using T = T64<N, K1>;
  constexpr int TX = T::TX, TY = T::TY, NT = T::NT, X1 = T::X1, Y1 = T::Y1, X2 = T::X2, Y2 = T::Y2;
  constexpr int R1 = X1 * Y1, R2 = X2 * Y2, FX = T::FX, NF = T::NF, JX = T::JX, NJ = T::NJ, L = N - 1;
  extern __shared__ __align__(16) double sm64[];
  double* const sphi = sm64 + T::o_phi;
  double* const smu = sm64 + T::o_mu;
  double* const sdp = sm64 + T::o_dp;
  double* const sface = sm64 + T::o_face;
  double* const sjat = sface;             // [K1][NJ]
  double* const ssob = sface + K1 * NJ;   // [N-1][X1][Y1]
  __shared__ uint8_t s_act[R1], s_cls[TX * TY];
  __shared__ uint16_t s_list[R1];
  __shared__ int s_n, s_bad;
  const int tid = threadIdx.x, lane = tid & 31, ti = tid / TY, tj = tid % TY;
  const int nty = (g.my + TY - 1) / TY;
  const double ix = c64.ix, iy = c64.iy, i2y = c64.i2y;
  const MulSpacing spacing = {ix, iy};

  gp_allow_dependents();
  gp_wait_for_earlier_kernels();
  const int ntile = *cnt;
  if (blockIdx.x == 0 && tid == 0) {
    *next_cnt = 0;  // the next step's list starts empty (read last by the step before)
    if (seen && *told != ntile) {  // the host's copy of the count (mapped memory), written when it changes
      *told = ntile;
      *reinterpret_cast<volatile int*>(seen) = ntile;
    }
  }
  {
#pragma unroll 1
    for (int q = blockIdx.x; q < ntile; q += gridDim.x) {
      const int t = list[q], x0 = (t / nty) * TX, y0 = (t % nty) * TY;
      __syncthreads();  // the previous tile's shared state has been read
      if (tid == 0) s_n = s_bad = 0;
#pragma unroll 1
      for (int e = tid; e < R2; e += NT) {
        const int i = e / Y2, j = e % Y2;
        const double* p = phi + (int64_t)gp_map_any(x0 - 2 + i, g.mx, g.bc.phi_x) * g.pitch + gp_map_any(y0 - 2 + j, g.my, g.bc.phi_y);
#pragma unroll
        for (int a = 0; a < N; a++) copy8(sphi + a * R2 + e, p + a * g.plane);
      }
#pragma unroll 1
      for (int e = tid; e < R1; e += NT) {
        const int i = e / Y1, j = e % Y1;
        const double* p = mu + (int64_t)gp_map_any(x0 - 1 + i, g.mx, g.bc.mu_x) * g.pitch + gp_map_any(y0 - 1 + j, g.my, g.bc.mu_y);
#pragma unroll
        for (int k = 0; k < K1; k++) copy8(smu + k * R1 + e, p + k * g.plane);
      }
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();

      // ring cells whose 3x3 phi block is flat (flat_block): Delta-phi +0; the others are listed
#pragma unroll 1
      for (int e0 = 0; e0 < R1; e0 += NT) {
        const int e = e0 + tid;
        bool act = false;
        if (e < R1) {
          const int i = e / Y1, j = e % Y1;
          if (x0 - 1 + i <= g.mx && y0 - 1 + j <= g.my) {
            bool flat = true;
#pragma unroll T::unroll
            for (int a = 0; a < N; a++) {
              const double* p = sphi + a * R2 + i * Y2 + j;
              const double c = p[Y2 + 1];
              bool f = (c >= 0.0) & (c <= 1.0);
#pragma unroll
              for (int di = 0; di < 3; di++)
#pragma unroll
                for (int dj = 0; dj < 3; dj++) f &= p[di * Y2 + dj] == c;
              flat &= f;
            }
            act = !flat;
          }
          s_act[e] = act;
#pragma unroll
          for (int a = 0; a < N; a++) sdp[a * R1 + e] = 0.0;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, act);
        int base = 0;
        if (lane == 0 && bal) base = atomicAdd(&s_n, __popc(bal));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (act) s_list[base + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)e;
      }
      __syncthreads();
      const int nact = s_n;

      // Gradient-energy terms of the faces next to a listed cell, per pair a < b: A = a_c^2 Q_n and
      // B = a_c |q|^2 (R^-1 da_c/dq)_n (anisotropic), A = Q_n (isotropic); function_A_01.h:101-219.
      // Face f: x-faces between rows i and i + 1 (of tile +- 2) at column j, then y-faces between
      // columns j and j + 1 at row i; sn, st: strides along and across its normal.
#pragma unroll 1
      for (int e = tid; nact && e < T::P * NF; e += NT) {
        const int p = T::P == 1 ? 0 : e / NF, f = T::P == 1 ? e : e % NF;
        const bool xf = f < FX;
        const int r = xf ? f : f - FX, w = xf ? Y1 : TY + 3;
        const int i = r / w + (xf ? 0 : 1), j = r % w + (xf ? 1 : 0);
        const int lo = (i - 1) * Y1 + j - 1, hi = xf ? lo + Y1 : lo + 1;  // the two cells' ring positions
        const bool in_lo = xf ? i >= 1 : j >= 1, in_hi = xf ? i <= TX + 1 : j <= TY + 1;
        if (!((in_lo && s_act[lo]) || (in_hi && s_act[hi]))) continue;
        int a = 0, b = 1;
        if (N > 2) pair_of<N>(p, a, b);
        const int sn = xf ? Y2 : 1, st = xf ? 1 : Y2;
        const double* const pa = sphi + a * R2 + i * Y2 + j;
        const double* const pb = sphi + b * R2 + i * Y2 + j;
        const double h = xf ? ix : iy;
        const double sa = 0.5 * (pa[sn] + pa[0]), sb = 0.5 * (pb[sn] + pb[0]);
        const double ga = (pa[sn] - pa[0]) * h, gb = (pb[sn] - pb[0]) * h;
        const double Qn = (sa * gb - sb * ga);
        double A = Qn, B = 0.0;
        if (m.anisotropy) {
          auto tang = [&](const double* v) {
            return xf ? (v[st] - v[-st]) * i2y : 0.5 * ((v[st] - v[0]) * ix + (v[0] - v[-st]) * ix);
          };
          const double Qt = 0.5 * (sa * (tang(pb) + tang(pb + sn)) - sb * (tang(pa) + tang(pa + sn)));
          double q0, q1, e0, e1, r0, r1;
          mul2(m.R[a][b], xf ? Qn : Qt, xf ? Qt : Qn, q0, q1);
          double ac;
          aniso_both(m.dab[a][b], q0, q1, ac, e0, e1);
          const double ac2 = ac * ac;
          mul2(m.Rinv[a][b], e0, e1, r0, r1);
          const double q2 = q0 * q0 + q1 * q1;
          A = ac2 * Qn;
          B = ac * q2 * (xf ? r0 : r1);
        }
        sface[(2 * p) * NF + f] = A;
        sface[(2 * p + 1) * NF + f] = B;
      }
      __syncthreads();

      // divphi of phase a at the ring cell whose phi is at p
      auto div_of = [&](const double* p) {
        const double c = p[0], gx = (p[Y2] - c) * ix, bgx = (c - p[-Y2]) * ix, gy = (p[1] - c) * iy, lgy = (c - p[-1]) * iy;
        double d = (gx - bgx) * ix;
        d += (gy - lgy) * iy;
        return d;
      };
      // lambda of every phase of the listed cells, an item each (calculate_divergence_phasefield.h:4-40)
#pragma unroll 1
      for (int it = tid; it < nact * N; it += NT) {
        const int cell = it / N, a = it - cell * N, e = s_list[cell], i1 = e / Y1, j1 = e % Y1;
        const double* const pc = sphi + (i1 + 1) * Y2 + j1 + 1;
        const double* const pp = pc + a * R2;
        if (!(fabs(div_of(pp)) > 0.0)) continue;  // its lambda stays 0
        double ph[N], divphi[N];
#pragma unroll
        for (int b = 0; b < N; b++) {
          ph[b] = pc[b * R2];
          divphi[b] = div_of(pc + b * R2);
        }
        const double pa = pp[0];
        const double cxa = 0.5 * ((pp[Y2] - pa) * ix + (pa - pp[-Y2]) * ix), cya = (pp[1] - pp[-1]) * i2y;
        // the face terms around the cell: front (back one row before), right (left one before)
        const double* const fx = sface + (i1 + 1) * Y1 + j1;
        const double* const fy = sface + FX + i1 * (TY + 3) + j1 + 1;
        double s1 = 0.0, s2 = 0.0, d1s = 0.0, d2s = 0.0;
#pragma unroll 1
        for (int b = 0; b < N; b++) {
          if (b == a) continue;
          const double* const pq = pc + b * R2;
          const double gam = m.Gamma[a][b], pb = pq[0];
          const double cxb = 0.5 * ((pq[Y2] - pb) * ix + (pb - pq[-Y2]) * ix), cyb = (pq[1] - pq[-1]) * i2y;
          const double Qcx = (pa * cxb - pb * cxa), Qcy = (pa * cyb - pb * cya);
          const int o = (a < b ? pair_index<N>(a, b) : pair_index<N>(b, a)) * 2 * NF, oB = o + NF;
          const double sg = a < b ? 1.0 : -1.0;
          const double sf = 0.5 * (pq[Y2] + pb), sb = 0.5 * (pb + pq[-Y2]), sr = 0.5 * (pq[1] + pb), sl = 0.5 * (pb + pq[-1]);
          double e1 = (((sg * fx[o]) * (-sf)) - ((sg * fx[o - Y1]) * (-sb))) * ix;
          e1 += (((sg * fy[o]) * (-sr)) - ((sg * fy[o - 1]) * (-sl))) * iy;
          e1 *= gam;
          d1s += e1;
          if (!m.anisotropy) {
            double sp = 0.0;
            sp += Qcx * cxb;
            sp += Qcy * cyb;
            sp *= gam;
            s1 += sp;
            continue;
          }
          double q0, q1, d0, d1, r0, r1;
          mul2(m.R[a][b], Qcx, Qcy, q0, q1);
          double ac1;
          aniso_both(m.dab[a][b], q0, q1, ac1, d0, d1);
          const double q2 = (q0 * q0 + q1 * q1);
          const double ac2 = ac1 * ac1;
          mul2(m.R[a][b], cxb, cyb, r0, r1);
          double sp1 = 0.0, sp2 = 0.0;
          sp1 += q0 * r0;
          sp1 += q1 * r1;
          sp2 += (d0)*r0;
          sp2 += (d1)*r1;
          sp1 *= gam * ac2;
          sp2 *= gam * ac1 * q2;
          s1 += sp1;
          s2 += sp2;
          double e2 = ((sg * fx[oB]) * (-sf) - (sg * fx[oB - Y1]) * (-sb)) * ix;
          e2 += ((sg * fy[oB]) * (-sr) - (sg * fy[oB - 1]) * (-sl)) * iy;
          e2 *= gam;
          d2s += e2;
        }
        double tt;
        if (!m.anisotropy) {
          const double dA = 2.0 * s1, divA = 2.0 * d1s;
          tt = -dA + divA;
        } else {
          const double dA = 2.0 * (s1 + s2), divA = (2.0 * (d1s + d2s) + 0.0);
          tt = -dA + divA;
        }
        double muc[K1], ds = 0.0;
#pragma unroll
        for (int k = 0; k < K1; k++) muc[k] = smu[k * R1 + e];
        const Th th = th_row(m, g, y0 - 1 + j1, g.t_linear);
#pragma unroll 1
        for (int b = 0; b < N; b++) {
          double c[K1];
          double psi = 0.0;
#pragma unroll
          for (int k = 0; k < K1; k++) {
            c[k] = c_mu<K1>(m, th, muc, b, k);
            psi -= muc[k] * c[k];
          }
          psi += free_energy<N, K1>(m, th, c, b);
          ds += psi * dhphi<N>(ph, pc[b * R2], pa, b, a);
        }
        sdp[a * R1 + e] = m.epsilon * (tt)-m.inv_eps * dwdphi<N>(m, ph, divphi, pa, a) - ds;
      }
      __syncthreads();
      // Delta-phi of the listed cells (calculate_divergence_phasefield.h:41-62, simplex_projection.h:1-49)
#pragma unroll 1
      for (int idx = tid; idx < nact; idx += NT) {
        const int e = s_list[idx];
        const double* const pc = sphi + (e / Y1 + 1) * Y2 + e % Y1 + 1;
        double ph[N], divphi[N], lambda[N], dp[N], sum_lambda = 0.0;
        int active = 0;
#pragma unroll
        for (int a = 0; a < N; a++) {
          ph[a] = pc[a * R2];
          divphi[a] = div_of(pc + a * R2);
          lambda[a] = sdp[a * R1 + e];
          if (fabs(divphi[a]) > 0.0) {
            sum_lambda += lambda[a];
            active++;
          }
        }
        if (N == 2) sum_lambda = active == 2 ? sum_lambda * 0.5 : sum_lambda;
        else if (active) sum_lambda = gp_ddiv(sum_lambda, (double)active);
        const double te = tau_phi<N>(m, ph) * m.epsilon, yte = 1.0 / te;
#pragma unroll
        for (int a = 0; a < N; a++) dp[a] = fabs(divphi[a]) > 0.0 ? quot(m.dt * (lambda[a] - sum_lambda), te, yte) : 0.0;
        project_simplex<N>(ph, divphi, dp);
#pragma unroll
        for (int a = 0; a < N; a++) sdp[a * R1 + e] = dp[a];
      }
      // s(phi) of the antitrapping term (obstacle), a ring cell and solid phase per item
      if (m.obstacle) {
#pragma unroll 1
        for (int it = tid; nact && it < L * R1; it += NT) {
          const int a = L == 1 ? 0 : it / R1, e = L == 1 ? it : it % R1;
          const double* const pc = sphi + (e / Y1 + 1) * Y2 + e % Y1 + 1;
          double ph[N];
#pragma unroll
          for (int b = 0; b < N; b++) ph[b] = pc[b * R2];
          const double pa = pc[a * R2];
          double s1 = 0.0, h = 3.0 * pa * pa - 2.0 * pa * pa * pa;  // hphi
#pragma unroll
          for (int b = 0; b < N; b++)
#pragma unroll
            for (int c = b + 1; c < N; c++)
              if (b != a && c != a) s1 += ph[b] * ph[c];
          s1 *= 2.0 * pa;
          h = h + s1;
          double s = 0.0;
          if (pa * (1.0 - pa) > 0.0) s = pa * (1.0 - h) / (sqrt(pa * (1.0 - pa)));
          ssob[it] = s;
        }
      }
      __syncthreads();

      // antitrapping currents of the tile's faces next to a listed cell (calculate_fluxes_concentration.h:4-145)
#pragma unroll 1
      for (int f = tid; nact && f < NJ; f += NT) {
        const bool xf = f < JX;
        const int r = xf ? f : f - JX, w = xf ? TY : TY + 1;
        const int ic = r / w + (xf ? 0 : 1), jc = r % w + (xf ? 1 : 0);  // the lower cell's ring position
        const int ec = ic * Y1 + jc, en = xf ? ec + Y1 : ec + 1;
        if (!s_act[ec] && !s_act[en]) continue;
        const int sn = xf ? Y2 : 1, st = xf ? 1 : Y2;
        const double* const pc = sphi + (ic + 1) * Y2 + jc + 1;
        const double h = xf ? ix : iy;
        auto tang = [&](const double* v) {
          return xf ? (v[st] - v[-st]) * i2y : 0.5 * ((v[st] - v[0]) * ix + (v[0] - v[-st]) * ix);
        };
        const double* const pl = pc + L * R2;
        const double gl = (pl[sn] - pl[0]) * h;
        const double tl = 0.5 * (tang(pl) + tang(pl + sn));
        const double norm_l = sqrt(tl * tl + gl * gl);
        const int y = y0 - 1 + jc;  // the lower cell's row; the face of ghosted row MESH_Y-2 carries none
        const bool skip = !xf && ((y + 3 == g.my - 2) || (y + 3 == 0));
        const Th th_c = th_row(m, g, y, false), th_n = xf ? th_c : th_row(m, g, y + 1, false);
        double j[K1], uc[K1], un[K1];
#pragma unroll
        for (int k = 0; k < K1; k++) {
          j[k] = 0.0;
          uc[k] = smu[k * R1 + ec];
          un[k] = smu[k * R1 + en];
        }
#pragma unroll 1
        for (int a = 0; a < L; a++) {
          const double* const pa = pc + a * R2;
          const double ga = (pa[sn] - pa[0]) * h;
          const double ta = 0.5 * (tang(pa) + tang(pa + sn));
          const double normg = sqrt(ta * ta + ga * ga);
          if (normg == 0.0 || skip) continue;
          double sp = ga * gl;
          sp += ta * tl;
          if (norm_l > 0.0) sp /= (norm_l * normg);
          const double dn = sdp[a * R1 + en], dc = sdp[a * R1 + ec];
#pragma unroll
          for (int k = 0; k < K1; k++) {
            const double cl_n = c_mu<K1>(m, th_n, un, L, k), cl_c = c_mu<K1>(m, th_c, uc, L, k);
            const double cs_n = c_mu<K1>(m, th_n, un, a, k), cs_c = c_mu<K1>(m, th_c, uc, a, k);
            const double fk = c64.atf[a][k];
            double v;
            if (m.obstacle)
              v = fk * fabs(sp) * 0.5 * (ssob[a * R1 + en] * (cl_n - cs_n) * dn + ssob[a * R1 + ec] * (cl_c - cs_c) * dc) * ga;
            else
              v = fk * fabs(sp) * m.s_well * ((cl_n - cs_n) * dn + (cl_c - cs_c) * dc) * ga;
            j[k] += v / normg;
          }
        }
#pragma unroll
        for (int k = 0; k < K1; k++) sjat[k * NJ + f] = j[k];
      }
      __syncthreads();

      // mu and phi of the tile (calculate_divergence_concentration.h:4-153)
      const int x = x0 + ti, y = y0 + tj, e = (ti + 1) * Y1 + tj + 1;
      if (ti < TX && x < g.mx && y < g.my) {
        const double* const pc = sphi + (ti + 2) * Y2 + tj + 2;
        double ph[N], phb[N], phf[N], phl[N], phr[N], Dc[N], U0[5][K1], jt[4][K1];
#pragma unroll
        for (int a = 0; a < N; a++) {
          ph[a] = pc[a * R2];
          phb[a] = pc[a * R2 - Y2];
          phf[a] = pc[a * R2 + Y2];
          phl[a] = pc[a * R2 - 1];
          phr[a] = pc[a * R2 + 1];
          Dc[a] = sdp[a * R1 + e];
        }
        const bool act = s_act[e];  // a flat cell carries no current on any face
        const int fx = ti * TY + tj, fy = JX + ti * (TY + 1) + tj;
#pragma unroll
        for (int k = 0; k < K1; k++) {
          const double* const u = smu + k * R1 + e;
          U0[0][k] = u[0];
          U0[1][k] = u[-Y1];
          U0[2][k] = u[Y1];
          U0[3][k] = u[-1];
          U0[4][k] = u[1];
          const double* const jk = sjat + k * NJ;
          jt[0][k] = act ? jk[fx + TY] : 0.0;
          jt[1][k] = act ? jk[fx] : 0.0;
          jt[2][k] = act ? jk[fy + 1] : 0.0;
          jt[3][k] = act ? jk[fy] : 0.0;
        }
        double mnew[K1];
        int one = -1;  // a flat cell of one pure phase
        bool pure = !act;
#pragma unroll
        for (int a = 0; a < N; a++) {
          if (ph[a] == 1.0 && one < 0) one = a;
          else pure = pure && ph[a] == 0.0;
        }
        if (pure && one >= 0)
          pure_cell<N, K1>(m, c64, th_row(m, g, y, false), one, U0, mnew);
        else
          cell_update<N, K1, false>(m, spacing, th_row(m, g, y, false), ph, phb, phf, phl, phr, U0[0], U0[1], U0[2], U0[3],
                                    U0[4], Dc, jt[0], jt[1], jt[2], jt[3], mnew);
        const int64_t o = (int64_t)x * g.pitch + y;
#pragma unroll
        for (int k = 0; k < K1; k++) mu_out[o + k * g.plane] = mnew[k];
        int hot = -1;
        bool onehot = true;
#pragma unroll
        for (int a = 0; a < N; a++) {
          const double v = ph[a] + Dc[a];
          phi_out[o + a * g.plane] = v;
          if (v == 1.0 && hot < 0) hot = a;
          else if (__double_as_longlong(v) != 0) onehot = false;  // -0 is not the pure field's +0
        }
        s_cls[tid] = onehot && hot >= 0 ? (uint8_t)hot : (uint8_t)0xFF;
      }
      __syncthreads();
      // purity word of the output tile (whole tile, first/last two rows, first/last two columns)
      const int ex = min(TX, g.mx - x0), ey = min(TY, g.my - y0);
      const int r0 = s_cls[0], rxh = s_cls[(ex - 1) * TY], ryh = s_cls[ey - 1];
      unsigned bad = 0u;
      if (ti < ex && tj < ey) bad = part_bits(ti, tj, ex, ey, s_cls[tid], r0, rxh, ryh);
      bad = __reduce_or_sync(0xffffffffu, bad);
      if (lane == 0 && bad) atomicOr(&s_bad, (int)bad);
      __syncthreads();
      if (tid == 0) wout[t] = word_of((uint32_t)s_bad, r0, rxh, ryh);
    }
  }
}

template <int N, int K1, bool SMOOTH>
cudaError_t launch_step(const gp_model& m, const Geo& g, const double* phi, const double* mu, double* dphi,
                        double* phi_out, double* mu_out, cudaStream_t s) {
  const dim3 blk(32, 8);
  const dim3 grd_r((g.my + 2 + 31) / 32, (g.mx + 2 + 7) / 8);
  k_dphi<N, K1, SMOOTH><<<grd_r, blk, 0, s>>>(m, g, phi, mu, dphi);
  const dim3 grd((g.my + 31) / 32, (g.mx + 7) / 8);
  Geo gu = g;
  gu.gov = nullptr;  // the concentration half step reads refreshed ghosts
  k_update<N, K1, SMOOTH><<<grd, blk, 0, s>>>(m, gu, phi, mu, dphi, phi_out, mu_out);
  return cudaGetLastError();
}

}  // namespace

static Geo make_geo(const gp_model& m, int pitch, int64_t plane, int rpitch, int64_t rplane, const gp_temp_step* temp,
                    const double* ghost_rows) {
  Geo g;
  g.noniso = m.nonisothermal ? 1 : 0;
  g.t_linear = temp ? temp->linear : 0;
  g.bc_t = m.bc_T[3];
  g.t_bottom = temp ? temp->bottom : 0.0;
  g.t_grad = temp ? temp->grad : 0.0;
  g.mx = (int)m.mesh_x;
  g.my = (int)m.mesh_y;
  g.pitch = pitch;
  g.plane = plane;
  g.rpitch = rpitch;
  g.rplane = rplane;
  g.bc = gp_bc_of(m);
  g.gov = ghost_rows;
  return g;
}

#define GP_ALL_CASES                                        \
  GP_CASE(2, 1) GP_CASE(2, 2) GP_CASE(2, 3)                 \
  GP_CASE(3, 1) GP_CASE(3, 2) GP_CASE(3, 3)                 \
  GP_CASE(4, 1) GP_CASE(4, 2) GP_CASE(4, 3)                 \
  GP_CASE(5, 1) GP_CASE(5, 2) GP_CASE(5, 3)                 \
  GP_CASE(6, 1) GP_CASE(6, 2) GP_CASE(6, 3)

// The tiles of a grid stepped by k_step64: static facts, purity words of the two state buffers.
struct gp_f64_tiles {
  C64 c;
  uint32_t* geo = nullptr;    // [n]
  uint32_t* words = nullptr;  // [2][n]
  int* list = nullptr;        // [n] tiles of the current step for k_step64, its two alternating counts, the count last
                              // told to the host
  int* seen = nullptr;        // that count in page-locked memory: read without waiting for the device, so it lags
  int n = 0, grid = 0;
  int dense_from = INT32_MAX;  // more listed tiles than this: the ring-array kernels are faster
};

// Page-locked words that a kernel writes and the host reads without waiting, one per context that needs one.
// Allocating page-locked memory takes 1 to 3 ms, longer than the rest of a small context, so the process keeps
// one page of them from the first such context on; contexts beyond its 1,024 words do without (they stay on
// the tile kernels).  The page is asked about before it is used again: a device reset takes it away.
static std::mutex word_lock;
static int* word_page = nullptr;
static bool word_used[1024];

static int* word_acquire() {
  const std::lock_guard<std::mutex> lock(word_lock);
  cudaPointerAttributes at;
  if (!word_page || cudaPointerGetAttributes(&at, word_page) != cudaSuccess || at.type != cudaMemoryTypeHost) {
    cudaGetLastError();
    word_page = nullptr;
    memset(word_used, 0, sizeof word_used);
    if (cudaHostAlloc((void**)&word_page, sizeof word_used / sizeof word_used[0] * sizeof(int),
                      cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      word_page = nullptr;
      return nullptr;
    }
  }
  for (size_t i = 0; i < sizeof word_used / sizeof word_used[0]; i++)
    if (!word_used[i]) {
      word_used[i] = true;
      word_page[i] = 0;
      return word_page + i;
    }
  return nullptr;
}

static void word_release(int* w) {
  const std::lock_guard<std::mutex> lock(word_lock);
  if (w && word_page && w >= word_page && w < word_page + sizeof word_used / sizeof word_used[0]) word_used[w - word_page] = false;
}

// The caller has waited for the kernels that use the tables.
void gp_f64_tiles_destroy(gp_f64_tiles* t) {
  if (!t) return;
  cudaFree(t->geo);
  cudaFree(t->words);
  cudaFree(t->list);
  word_release(t->seen);
  delete t;
}

static bool power_of_two(double d) {
  int e;
  return frexp(d, &e) == 0.5 && e > -500 && e < 500;
}

// Whether k_step64 takes the model: it evaluates a pair's terms once for both of its phases, and
// multiplies by the spacings' reciprocals.
static bool tile_model(const gp_model& m) {
  if (!power_of_two(m.dx) || !power_of_two(m.dy)) return false;
  for (int a = 0; a < m.N; a++)
    for (int b = a + 1; b < m.N; b++) {
      if (!(m.Gamma[a][b] == m.Gamma[b][a]) || !(m.dab[a][b] == m.dab[b][a])) return false;
      for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++)
          if (!(m.R[a][b][i][j] == m.R[b][a][i][j]) || !(m.Rinv[a][b][i][j] == m.Rinv[b][a][i][j])) return false;
    }
  return true;
}

// *out stays nullptr for a model the tile kernel does not take.  The fills run on the legacy stream: the caller waits
// for them before it uses another one.
cudaError_t gp_f64_tiles_create(const gp_model& m, gp_f64_tiles** out) {
  *out = nullptr;
  if (!tile_model(m)) return cudaSuccess;
  constexpr int TX = T64<2, 1>::TX, TY = T64<2, 1>::TY;
  const int64_t n = ((m.mesh_x + TX - 1) / TX) * ((m.mesh_y + TY - 1) / TY);
  if (n > INT32_MAX / 8) return cudaSuccess;
  int dev = 0, sms = 0, occ = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
#define GP_CASE(NN, KK)                                                                                           \
  if (m.N == NN && m.K1 == KK) {                                                                                  \
    if (e == cudaSuccess)                                                                                         \
      e = cudaFuncSetAttribute(k_step64<NN, KK>, cudaFuncAttributeMaxDynamicSharedMemorySize,                     \
                               (int)T64<NN, KK>::bytes);                                                          \
    if (e == cudaSuccess)                                                                                         \
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_step64<NN, KK>, T64<NN, KK>::NT, T64<NN, KK>::bytes); \
  }
  GP_ALL_CASES
#undef GP_CASE
  if (e != cudaSuccess) return e;
  gp_f64_tiles* t = new gp_f64_tiles();
  t->n = (int)n;
  memset(&t->c, 0, sizeof t->c);
  t->c.ix = 1.0 / m.dx;
  t->c.iy = 1.0 / m.dy;
  t->c.i2y = 1.0 / (2.0 * m.dy);
  for (int a = 0; a < m.N; a++)
    for (int i = 0; i < m.K1; i++) {
      t->c.atf[a][i] = (1.0 - m.Diff[a][i][i] / m.Diff[m.N - 1][i][i]);
      for (int j = 0; j < m.K1; j++) {
        volatile double s = 0.0;  // each product and sum rounded, as the kernels do
        for (int b = 0; b < m.N; b++)
          for (int k = 0; k < m.K1; k++) {
            volatile double v = m.Diff[b][i][k] * m.cmu[b][k][j];
            v = v * (a == b ? 1.0 : 0.0);
            s = s + v;
          }
        t->c.Dp[a][i][j] = s;
      }
    }
  const int most = sms * (occ > 0 ? occ : 1);
  t->grid = t->n < most ? t->n : most;
  // Two phases: a listed tile costs more than its share of k_dphi and k_update (its ring is 1.4 times its cells,
  // and two blocks an SM overlap less than their three), so they win where most tiles are listed, unless one
  // round of resident blocks takes them all.  us per step, tiles against ring array, listed / all: 200^2 obstacle
  // 247/325 19.8 and 25.7; 300x280 well 558/684 31.9 and 29.2, 684/684 40.3 and 29.1; 512^2 obstacle 776/2048 44.9
  // and 52.1, well 1012/2048 54.3 and 49.6, 1544/2048 73.6 and 57.9; 700^2 obstacle 1070/3872 63.3 and 67.5,
  // 1741/3872 88.5 and 88.0; 1024^2 well 2269/8192 102 and 110, 3474/8192 146 and 143, 5408/8192 219 and 189.
  // Three and four phases share more between the pairs and win at any density (four phases, all 3,425 of
  // 3,872 listed: 428 and 695).
  if (m.N == 2) t->dense_from = most > 2 * t->n / 5 ? most : 2 * t->n / 5;
  std::vector<uint32_t> geo(t->n);
  const gp_bc bc = gp_bc_of(m);
  for (int k = 0; k < t->n; k++) geo[k] = tile_geo((int)m.mesh_x, (int)m.mesh_y, bc, k, TX, TY);
  e = cudaMalloc(&t->geo, sizeof(uint32_t) * n);
  if (e == cudaSuccess) e = cudaMemcpy(t->geo, geo.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&t->words, 2 * sizeof(uint32_t) * n);
  if (e == cudaSuccess) e = cudaMemset(t->words, 0, 2 * sizeof(uint32_t) * n);
  if (e == cudaSuccess) e = cudaMalloc(&t->list, sizeof(int) * (n + 3));
  if (e == cudaSuccess) e = cudaMemset(t->list + n, 0, 3 * sizeof(int));
  if (e == cudaSuccess && t->dense_from < t->n) t->seen = word_acquire();
  if (e != cudaSuccess) {
    gp_f64_tiles_destroy(t);
    return e;
  }
  *out = t;
  return cudaSuccess;
}

// Nothing is known of the tiles, and both list counts start at 0 again (they alternate with the buffers).
cudaError_t gp_f64_tiles_invalidate(gp_f64_tiles* t, cudaStream_t s) {
  if (!t) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(t->words, 0, 2 * sizeof(uint32_t) * (size_t)t->n, s);
  return e == cudaSuccess ? cudaMemsetAsync(t->list + t->n, 0, 2 * sizeof(int), s) : e;
}

// The tables for the state in buffer parity p, from the state itself.
cudaError_t gp_f64_tiles_survey(const gp_model& m, gp_f64_tiles* t, int p, int pitch, int64_t plane, const double* phi,
                                cudaStream_t s) {
  const gp_temp_step none = {};
  const Geo g = make_geo(m, pitch, plane, 0, 0, &none, nullptr);
#define GP_CASE(NN, KK)                                                                                       \
  if (m.N == NN && m.K1 == KK) {                                                                              \
    k_words64<NN, KK><<<(t->n + 7) / 8, 256, 0, s>>>(g, phi, t->words + (size_t)p * t->n,                     \
                                                     t->words + (size_t)(p ^ 1) * t->n, t->list + t->n, t->n); \
    return cudaGetLastError();                                                                                \
  }
  GP_ALL_CASES
#undef GP_CASE
  return cudaErrorInvalidValue;
}

// Whether the last count the host has seen makes the ring-array kernels the faster ones.  Either path gives the
// same bits, so it does not matter that the count lags.
bool gp_f64_tiles_dense(const gp_f64_tiles* t) {
  return t->seen && *reinterpret_cast<volatile int*>(t->seen) > t->dense_from;
}

// The list of the step from buffer parity p is empty.  A step leaves the next parity's count at 0, which is
// enough while steps alternate; a caller's captured step may be replayed from one parity again and again, so
// there this goes first.
cudaError_t gp_f64_tiles_empty_list(gp_f64_tiles* t, int p, cudaStream_t s) {
  return cudaMemsetAsync(t->list + t->n + p, 0, sizeof(int), s);
}

// One step by the tile kernels from buffer parity p into the other: two launches.
cudaError_t gp_f64_step_tiled(const gp_model& m, gp_f64_tiles* t, int p, int pitch, int64_t plane, const double* phi,
                              const double* mu, double* phi_out, double* mu_out, cudaStream_t s,
                              const gp_temp_step* temp) {
  if (m.nonisothermal && !temp) return cudaErrorInvalidValue;
  const Geo g = make_geo(m, pitch, plane, 0, 0, temp, nullptr);
  const uint32_t* win = t->words + (size_t)p * t->n;
  uint32_t* wout = t->words + (size_t)(p ^ 1) * t->n;
  int *cnt = t->list + t->n + p, *next = t->list + t->n + (p ^ 1);
#define GP_CASE(NN, KK)                                                                                              \
  if (m.N == NN && m.K1 == KK) {                                                                                     \
    cudaError_t e = gp_launch_dependent(k_lean64<NN, KK>, (t->n + 7) / 8, 256, 0, s, m, t->c, g, t->geo, win, wout,     \
                                     t->n, mu, phi_out, mu_out, t->list, cnt);                                       \
    if (e == cudaSuccess)                                                                                            \
      e = gp_launch_dependent(k_step64<NN, KK>, t->grid, T64<NN, KK>::NT, T64<NN, KK>::bytes, s, m, t->c, g, wout, phi, \
                              mu, phi_out, mu_out, t->list, cnt, next, t->seen, t->list + t->n + 2);                 \
    return e;                                                                                                        \
  }
  GP_ALL_CASES
#undef GP_CASE
  return cudaErrorInvalidValue;
}

// Delta-phi of a state into the ring array alone (the tile kernel keeps its own in shared memory).
cudaError_t gp_f64_dphi(const gp_model& m, int pitch, int64_t plane, int rpitch, int64_t rplane, const double* phi,
                        const double* mu, double* dphi, cudaStream_t s, const gp_temp_step* temp) {
  if (m.nonisothermal && !temp) return cudaErrorInvalidValue;
  const Geo g = make_geo(m, pitch, plane, rpitch, rplane, temp, nullptr);
  const dim3 blk(32, 8), grd((g.my + 2 + 31) / 32, (g.mx + 2 + 7) / 8);
#define GP_CASE(NN, KK)                                                     \
  if (m.N == NN && m.K1 == KK) {                                            \
    k_dphi<NN, KK, false><<<grd, blk, 0, s>>>(m, g, phi, mu, dphi);         \
    return cudaGetLastError();                                              \
  }
  GP_ALL_CASES
#undef GP_CASE
  return cudaErrorInvalidValue;
}

// One step through the ring array: two launches.
cudaError_t gp_f64_step(const gp_model& m, int pitch, int64_t plane, int rpitch, int64_t rplane,
                        const double* phi, const double* mu, double* dphi, double* phi_out, double* mu_out,
                        cudaStream_t s, bool smooth, const double* ghost_rows, const gp_temp_step* temp) {
  if (m.nonisothermal && !temp) return cudaErrorInvalidValue;  // the step needs its temperature
  const Geo g = make_geo(m, pitch, plane, rpitch, rplane, temp, ghost_rows);
#define GP_CASE(NN, KK)                                                                           \
  if (m.N == NN && m.K1 == KK)                                                                    \
    return smooth ? launch_step<NN, KK, true>(m, g, phi, mu, dphi, phi_out, mu_out, s)            \
                  : launch_step<NN, KK, false>(m, g, phi, mu, dphi, phi_out, mu_out, s);
  GP_ALL_CASES
#undef GP_CASE
  return cudaErrorInvalidValue;
}
