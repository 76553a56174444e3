// gp_adjoint.cu -- hand-written adjoint of the explicit step (binary alloys:
// 2 phases, one independent chemical potential) with sqrt(N) checkpointing.
//
// Forward: the step of gp_adjoint_cell.cuh (the plain step's model) in the
// working precision T (float: the chosen form; double: the reference
// adjoint), one kernel per step: a block stages a tile, computes Delta-phi on
// the tile and one ring in shared memory, then the mu/phi update.  Every
// `every`-th state is kept (checkpoints).
//
// Reverse of one step n (state x_n, adjoint lambda_{n+1} of x_{n+1}).  The
// adjoint of a cell's flux divergences depends on its own phi and lambda_mu
// alone, so the dense part is a gather; only cells with phi gradients near
// them (listed when the segment is recomputed, a few percent of a grid) scatter:
//   1. k_rev_cell, every cell: reverse of its mu/phi update and of the
//      diffusion flux through its four faces (plain stores, one writer);
//   2. k_rev_jat, the faces of listed cells: reverse of the antitrapping
//      current, scattered by atomic adds into phi, mu and Delta-phi;
//   3. k_rev_dphi, the listed cells: reverse of Delta-phi, eight lanes per
//      cell, scattered into its 3x3 phi stencil and its mu.
// Ghost reads are boundary index maps, so their adjoints land on the mapped
// interior cells.  Parameter gradients accumulate in FP64 per block.
// Backward: segments of `every` steps, last first: the segment is recomputed
// from its checkpoint into a buffer of `every` states (each with its Delta-phi
// and its list), then reversed.
// Memory: ceil(N / every) + every states (every = ceil(sqrt(N)) by default), and for each state of a segment
// its Delta-phi and list, about as much as the state, or for one state at a time (Adj::reserve).

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "gp_common.cuh"
#include "gp_adjoint_cell.cuh"

extern "C" void gp_set_error(const char* fmt, ...);

namespace {

using namespace gpadj;

struct Geo {
  int mx, my, pitch, rpitch;
  int64_t plane, rplane;  // elements per state plane / Delta-phi ring plane
  gp_bc bc;
};

// state layout: planes phi_0, phi_1, mu, each [mx][pitch]
template <typename T>
__device__ __forceinline__ T ld_phi(const T* st, const Geo& g, int x, int y, int a) {
  return st[a * g.plane + (int64_t)gp_map(x, g.mx, g.bc.phi_x) * g.pitch + gp_map(y, g.my, g.bc.phi_y)];
}
template <typename T>
__device__ __forceinline__ T ld_mu(const T* st, const Geo& g, int x, int y) {
  return st[2 * g.plane + (int64_t)gp_map(x, g.mx, g.bc.mu_x) * g.pitch + gp_map(y, g.my, g.bc.mu_y)];
}
__device__ __forceinline__ int64_t ix_phi(const Geo& g, int x, int y, int a) {
  return a * g.plane + (int64_t)gp_map(x, g.mx, g.bc.phi_x) * g.pitch + gp_map(y, g.my, g.bc.phi_y);
}
__device__ __forceinline__ int64_t ix_mu(const Geo& g, int x, int y) {
  return 2 * g.plane + (int64_t)gp_map(x, g.mx, g.bc.mu_x) * g.pitch + gp_map(y, g.my, g.bc.mu_y);
}
// Delta-phi ring: cells x in [-1, mx], y in [-1, my]
__device__ __forceinline__ int64_t ix_ring(const Geo& g, int x, int y, int a) {
  return a * g.rplane + (int64_t)(x + 1) * g.rpitch + (y + 1);
}

template <typename T>
__device__ __forceinline__ void load_P(const T* st, const Geo& g, int x, int y, T (&P)[3][3][2]) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int a = 0; a < 2; a++) P[i][j][a] = ld_phi(st, g, x + i - 1, y + j - 1, a);
}

// The 3x3 block holds one value in [0, 1] per phase: every phi gradient is 0, no phase is active,
// Delta-phi is 0 whatever mu is, and no antitrapping current crosses the cell's faces.
template <typename T>
__device__ __forceinline__ bool flat_P(const T (&P)[3][3][2]) {
  bool f = true;
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const T c = P[1][1][a];
    f &= (c >= (T)0) & (c <= (T)1);  // no short circuit: a branch per compare costs more than the compares
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) f &= P[i][j][a] == c;
  }
  return f;
}

// Face k of interior cell (x, y): 0 = x+, 1 = x-, 2 = y+, 3 = y-; M[5], D[5]:
// mu and Delta-phi (phase 0) of the cell and its x-, x+, y-, y+ neighbours.
template <typename T, bool POW2>
__device__ __forceinline__ Face<T> cell_face(const AM<T, POW2>& m, const Geo& g, int y, const T (&P)[3][3][2],
                                             const T (&M)[5], const T (&D)[5], int k) {
  Face<T> f;
  auto cy = [&](int i, int a) { return m.qt(P[i][2][a] - P[i][0][a]); };
  auto cx = [&](int j, int a) { return (T)0.5 * (m.qx(P[2][j][a] - P[1][j][a]) + m.qx(P[1][j][a] - P[0][j][a])); };
  for (int a = 0; a < 2; a++) {
    if (k == 0) {
      f.pc[a] = P[1][1][a]; f.pn[a] = P[2][1][a]; f.tc[a] = cy(1, a); f.tn[a] = cy(2, a);
    } else if (k == 1) {
      f.pc[a] = P[0][1][a]; f.pn[a] = P[1][1][a]; f.tc[a] = cy(0, a); f.tn[a] = cy(1, a);
    } else if (k == 2) {
      f.pc[a] = P[1][1][a]; f.pn[a] = P[1][2][a]; f.tc[a] = cx(1, a); f.tn[a] = cx(2, a);
    } else {
      f.pc[a] = P[1][0][a]; f.pn[a] = P[1][1][a]; f.tc[a] = cx(0, a); f.tn[a] = cx(1, a);
    }
  }
  // neighbour slots: 0 centre, 1 x-, 2 x+, 3 y-, 4 y+
  const int cs = k == 1 ? 1 : (k == 3 ? 3 : 0), ns = k == 0 ? 2 : (k == 2 ? 4 : 0);
  f.muc = M[cs]; f.mun = M[ns];
  f.dpc = D[cs]; f.dpn = D[ns];
  f.h = (k >> 1) ? m.dy : m.dx;
  f.ih = (k >> 1) ? m.iy : m.ix;
  const int ylow = k == 3 ? y - 1 : y;  // the face's lower cell
  f.skip = (k >> 1) && (ylow + 3 == g.my - 2);
  return f;
}

// the diffusion flux of face k alone (fface on the cell's operands, without the antitrapping ones)
template <typename T, bool POW2>
__device__ __forceinline__ T cell_flux(const AM<T, POW2>& m, int dir, T pc0, T pc1, T pn0, T pn1, T muc,
                                       T mun) {
  const T Dc = m.Ds * m.cmu[0] * pc0 + m.Dl * m.cmu[1] * pc1;
  const T Dn = m.Ds * m.cmu[0] * pn0 + m.Dl * m.cmu[1] * pn1;
  return (Dn + Dc) * (T)0.5 * m.qd(dir, mun - muc);
}

// Start of a kernel launched as a dependent of the one before it: what its pointers lead to is written by
// kernels of the same chain, so none of them is `const __restrict__` (gp_common.cuh).
__device__ __forceinline__ void begin_dependent() {
  gp_allow_dependents();
  gp_wait_for_earlier_kernels();
}

// Block tile of the dense kernels: a cell per thread, y fastest (a warp per tile row).
constexpr int TX = 8, TY = 32, NT = TX * TY;
constexpr int X1 = TX + 2, Y1 = TY + 2, X2 = TX + 4, Y2 = TY + 4;

__device__ __forceinline__ void tile_origin(const Geo& g, int& x0, int& y0) {
  const int nty = (g.my + TY - 1) / TY;
  x0 = (int)(blockIdx.x / nty) * TX;
  y0 = (int)(blockIdx.x % nty) * TY;
}

// Ring position (x, y) = (x0 - 1 + i, y0 - 1 + j) of the tile belongs to it: one of its cells, or a
// cell of the grid's ghost ring beside it.
__device__ __forceinline__ bool owns_ring(const Geo& g, int x, int y, int i, int j) {
  return x <= g.mx && y <= g.my && ((i >= 1 && i <= TX) || x == -1 || (i == TX + 1 && x == g.mx)) &&
         ((j >= 1 && j <= TY) || y == -1 || (j == TY + 1 && y == g.my));
}

// ------------------------------------------------------------------ forward

// One step st -> out (out == nullptr: Delta-phi and the list only).  With ring: Delta-phi is also
// written there (interior and ghost ring), and the ring cells whose phi block is not flat are
// appended to list (as ring offsets), their number in *cnt.
// Bound by latency: a 512^2 FP32 step moves 6 MB within L2, and a block's chain is stage -> flags ->
// Delta-phi -> update.  Cells with a flat block (all but a few percent) skip the phase-field
// arithmetic; the others are compacted first, so that a warp of the tile does not wait for the few
// of its lanes that hold an interface.
// 18 us (ncu, 512^2 FP32, flushed caches) against about 50 for the two dense kernels before.
template <typename T, bool POW2>
__global__ void __launch_bounds__(NT) k_fwd(const __grid_constant__ AM<T, POW2> m, Geo g, const T* st, T* out, T* ring,
                                            int* list, int* cnt) {
  begin_dependent();
  __shared__ T sp[2][X2][Y2], su[X1][Y1], sd[2][X1][Y1];
  __shared__ int s_list[X1 * Y1], s_own[X1 * Y1], s_n, s_m, s_base;
  __shared__ uint8_t s_act[X1 * Y1];
  int x0, y0;
  tile_origin(g, x0, y0);
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) s_n = s_m = 0;
  for (int e = tid; e < X2 * Y2; e += NT) {
    const int i = e / Y2, j = e % Y2;
    const int64_t o = (int64_t)gp_map_any(x0 - 2 + i, g.mx, g.bc.phi_x) * g.pitch + gp_map_any(y0 - 2 + j, g.my, g.bc.phi_y);
    sp[0][i][j] = st[o];
    sp[1][i][j] = st[g.plane + o];
  }
  for (int e = tid; e < X1 * Y1; e += NT) {
    const int i = e / Y1, j = e % Y1;
    su[i][j] = st[2 * g.plane + (int64_t)gp_map_any(x0 - 1 + i, g.mx, g.bc.mu_x) * g.pitch +
                  gp_map_any(y0 - 1 + j, g.my, g.bc.mu_y)];
  }
  __syncthreads();
  auto block3 = [&](int i, int j, T (&P)[3][3][2]) {  // around ring position (i, j)
#pragma unroll
    for (int di = 0; di < 3; di++)
#pragma unroll
      for (int dj = 0; dj < 3; dj++)
#pragma unroll
        for (int a = 0; a < 2; a++) P[di][dj][a] = sp[a][i + di][j + dj];
  };
  for (int e0 = 0; e0 < X1 * Y1; e0 += NT) {
    const int e = e0 + tid;
    bool act = false, own = false;
    if (e < X1 * Y1) {
      const int i = e / Y1, j = e % Y1, x = x0 - 1 + i, y = y0 - 1 + j;
      sd[0][i][j] = sd[1][i][j] = (T)0;
      if (x <= g.mx && y <= g.my) {
        T P[3][3][2];
        block3(i, j, P);
        act = !flat_P(P);
        s_act[e] = act;
        own = act && ring && owns_ring(g, x, y, i, j);
      }
    }
    const unsigned below = (1u << lane) - 1u;
    const unsigned bal = __ballot_sync(0xffffffffu, act), balo = __ballot_sync(0xffffffffu, own);
    int base = 0, baseo = 0;
    if (lane == 0 && bal) base = atomicAdd(&s_n, __popc(bal));
    if (lane == 0 && balo) baseo = atomicAdd(&s_m, __popc(balo));
    base = __shfl_sync(0xffffffffu, base, 0);
    baseo = __shfl_sync(0xffffffffu, baseo, 0);
    if (act) s_list[base + __popc(bal & below)] = e;
    if (own) s_own[baseo + __popc(balo & below)] = e;
  }
  __syncthreads();
  if (ring && tid == 0 && s_m) s_base = atomicAdd(cnt, s_m);
  for (int q = tid; q < s_n; q += NT) {
    const int e = s_list[q], i = e / Y1, j = e % Y1;
    T P[3][3][2], dp[2];
    block3(i, j, P);
    dphi_fwd(m, P, su[i][j], dp);
    sd[0][i][j] = dp[0];
    sd[1][i][j] = dp[1];
  }
  __syncthreads();
  if (ring) {
    for (int q = tid; q < s_m; q += NT) {
      const int e = s_own[q];
      list[s_base + q] = (int)ix_ring(g, x0 - 1 + e / Y1, y0 - 1 + e % Y1, 0);
    }
    for (int e = tid; e < X1 * Y1; e += NT) {
      const int i = e / Y1, j = e % Y1, x = x0 - 1 + i, y = y0 - 1 + j;
      if (!owns_ring(g, x, y, i, j)) continue;
      ring[ix_ring(g, x, y, 0)] = sd[0][i][j];
      ring[ix_ring(g, x, y, 1)] = sd[1][i][j];
    }
  }
  const int i = tid / TY, j = tid % TY, x = x0 + i, y = y0 + j;
  if (!out || x >= g.mx || y >= g.my) return;
  T P[3][3][2], F[4], J[4];
  block3(i + 1, j + 1, P);
  const T M[5] = {su[i + 1][j + 1], su[i][j + 1], su[i + 2][j + 1], su[i + 1][j], su[i + 1][j + 2]};
  const T ph[2] = {P[1][1][0], P[1][1][1]};
  F[0] = cell_flux(m, 0, ph[0], ph[1], P[2][1][0], P[2][1][1], M[0], M[2]);
  F[1] = cell_flux(m, 0, P[0][1][0], P[0][1][1], ph[0], ph[1], M[1], M[0]);
  F[2] = cell_flux(m, 1, ph[0], ph[1], P[1][2][0], P[1][2][1], M[0], M[4]);
  F[3] = cell_flux(m, 1, P[1][0][0], P[1][0][1], ph[0], ph[1], M[3], M[0]);
  const T Dc[2] = {sd[0][i + 1][j + 1], sd[1][i + 1][j + 1]};
#pragma unroll
  for (int k = 0; k < 4; k++) J[k] = (T)0;
  if (s_act[(i + 1) * Y1 + j + 1]) {
    const T D[5] = {Dc[0], sd[0][i][j + 1], sd[0][i + 2][j + 1], sd[0][i + 1][j], sd[0][i + 1][j + 2]};
#pragma unroll
    for (int k = 0; k < 4; k++) J[k] = jface(m, cell_face(m, g, y, P, M, D, k));
  }
  const int64_t o = (int64_t)x * g.pitch + y;
  out[2 * g.plane + o] = mu_new(m, ph, M[0], Dc, F, J);
  out[o] = ph[0] + Dc[0];
  out[g.plane + o] = ph[1] + Dc[1];
}

// ------------------------------------------------------------------ reverse

// Adjoint of a cell's divflux (gdf) over dt: d mu_new / d c times lambda_mu (mu_new_rev); that of
// divjat is its negative.
template <typename T, bool POW2>
__device__ __forceinline__ T cell_ldc(const AM<T, POW2>& m, T p0, T p1, T lmn) {
  if (p0 == (T)1) return (T)2 * m.A[0] * lmn;
  if (p1 == (T)1) return (T)2 * m.A[1] * lmn;
  return lmn / (m.cmu[0] * hfun(p0) + m.cmu[1] * hfun(p1));
}

// Sum of v over the block into *slot (its only writer; launches that share it are ordered).
__device__ __forceinline__ void block_add(double v, double* slot) {
  __shared__ double s[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();  // s of a previous call has been read
  if (lane == 0) s[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < nw; i++) t += s[i];
    if (t != 0.0) *slot += t;
  }
}

// 1. reverse of the cell update and of the diffusion fluxes: every contribution that reaches a
// cell's own phi and mu through its update and its four faces, gathered (a boundary cell also takes
// the ghost cell that maps to it).  Writes lam_out and the cell's Delta-phi adjoint (ldphi; 0 on the
// ghost ring).  part[block] accumulates the D_liquid gradient, each face counted by its lower cell.
// Bound by its loads: 6 planes in, 5 out, with one synchronisation.
template <typename T, bool POW2>
__global__ void __launch_bounds__(NT) k_rev_cell(const __grid_constant__ AM<T, POW2> m, Geo g, const T* st, const T* ring,
                                                 const T* lam_in, T* lam_out, T* ldphi, double* part) {
  begin_dependent();
  __shared__ T sp[2][X1][Y1], su[X1][Y1], sg[X1][Y1];
  int x0, y0;
  tile_origin(g, x0, y0);
  const int tid = threadIdx.x;
  const T* const lmu_in = lam_in + 2 * g.plane;
  for (int e = tid; e < X1 * Y1; e += NT) {
    const int i = e / Y1, j = e % Y1, x = x0 - 1 + i, y = y0 - 1 + j;
    const int64_t o = (int64_t)gp_map_any(x, g.mx, g.bc.phi_x) * g.pitch + gp_map_any(y, g.my, g.bc.phi_y);
    const T p0 = st[o], p1 = st[g.plane + o];
    sp[0][i][j] = p0;
    sp[1][i][j] = p1;
    su[i][j] = st[2 * g.plane + (int64_t)gp_map_any(x, g.mx, g.bc.mu_x) * g.pitch + gp_map_any(y, g.my, g.bc.mu_y)];
    const bool in = x >= 0 && x < g.mx && y >= 0 && y < g.my;
    sg[i][j] = in ? cell_ldc(m, p0, p1, lmu_in[(int64_t)x * g.pitch + y]) * m.dt : (T)0;
    if (!in && owns_ring(g, x, y, i, j)) ldphi[ix_ring(g, x, y, 0)] = ldphi[ix_ring(g, x, y, 1)] = (T)0;
  }
  __syncthreads();
  double dl = 0.0;
  const int i = tid / TY + 1, j = tid % TY + 1, x = x0 + i - 1, y = y0 + j - 1;
  if (x < g.mx && y < g.my) {
    const int64_t o = (int64_t)x * g.pitch + y;
    const T ph[2] = {sp[0][i][j], sp[1][i][j]};
    const T M[5] = {su[i][j], su[i - 1][j], su[i + 1][j], su[i][j - 1], su[i][j + 1]};
    const T lp0 = lam_in[o], lp1 = lam_in[g.plane + o], lmn = lmu_in[o];
    T lph[2] = {lp0, lp1}, lmu = (T)0, ldp[2] = {lp0, lp1};
    if (ph[0] == (T)1 || ph[1] == (T)1) {
      const int b = ph[0] == (T)1 ? 0 : 1;
      lmu = (T)2 * m.A[b] * lmn * m.cmu[b];
    } else {
      T P[3][3][2], F[4], J[4], df, dj;
#pragma unroll
      for (int di = 0; di < 3; di++)
#pragma unroll
        for (int dj2 = 0; dj2 < 3; dj2++)
#pragma unroll
          for (int a = 0; a < 2; a++) P[di][dj2][a] = sp[a][i - 1 + di][j - 1 + dj2];
      T D[5];
      const T* r = ring + ix_ring(g, x, y, 0);
      D[0] = r[0];
      D[1] = r[-g.rpitch];
      D[2] = r[g.rpitch];
      D[3] = r[-1];
      D[4] = r[1];
      const T Dc[2] = {D[0], r[g.rplane]};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const Face<T> f = cell_face(m, g, y, P, M, D, k);
        F[k] = fface(m, f);
        J[k] = jface(m, f);
      }
      mu_new_rev(m, ph, M[0], Dc, F, J, lmn, lph, lmu, ldp, df, dj);
    }
    ldphi[ix_ring(g, x, y, 0)] = ldp[0];
    ldphi[ix_ring(g, x, y, 1)] = ldp[1];
    // the diffusion fluxes: s = +1 where the cell is the face's lower one
    const T k0 = m.Ds * m.cmu[0], k1 = m.Dl * m.cmu[1];
    const T Dme = k0 * ph[0] + k1 * ph[1];
    T sD = (T)0, sM = (T)0;  // summed apart: one rounding at the scale of the adjoint they are added to
    // p1: the two cells' phase 1, for the D_liquid gradient that is returned
    auto gather = [&](T s, T g_lo, T g_hi, T mu_lo, T mu_hi, T Dsum, T p1, int dir, bool to_phi, bool to_mu) {
      const T lF = m.qd(dir, g_lo - g_hi);
      T lD, lg;
      flux_rev(m.qd(dir, mu_hi - mu_lo), Dsum, lF, lD, lg);
      if (to_phi) sD += lD;
      if (to_mu) sM -= s * m.qd(dir, lg);
      return lF != (T)0 ? (double)(lD * m.cmu[1] * p1) : 0.0;
    };
    const T gme = sg[i][j];
    auto nb = [&](int a, int ii, int jj) { return sp[a][ii][jj]; };
    auto Dnb = [&](int ii, int jj) { return k0 * nb(0, ii, jj) + k1 * nb(1, ii, jj); };
    const double a0 = gather((T)1, gme, sg[i + 1][j], M[0], M[2], Dnb(i + 1, j) + Dme, ph[1] + nb(1, i + 1, j), 0, true, true);
    const double a1 = gather((T)-1, sg[i - 1][j], gme, M[1], M[0], Dme + Dnb(i - 1, j), nb(1, i - 1, j) + ph[1], 0, true, true);
    const double a2 = gather((T)1, gme, sg[i][j + 1], M[0], M[4], Dnb(i, j + 1) + Dme, ph[1] + nb(1, i, j + 1), 1, true, true);
    const double a3 = gather((T)-1, sg[i][j - 1], gme, M[3], M[0], Dme + Dnb(i, j - 1), nb(1, i, j - 1) + ph[1], 1, true, true);
    dl += a0 + a2;  // each face by its lower cell; the grid's first ones by their upper
    if (x == 0) dl += a1;
    if (y == 0) dl += a3;
    // the ghost cell (ghost row -1 or M, against the grid's first or last row `e`) that maps to this one
    auto ghost = [&](bool along_x, bool low) {
      const int Mg = along_x ? g.mx : g.my, v = low ? -1 : Mg, e = low ? 0 : Mg - 1, own = along_x ? x : y;
      const int mp = gp_map(v, Mg, along_x ? g.bc.phi_x : g.bc.phi_y), mm = gp_map(v, Mg, along_x ? g.bc.mu_x : g.bc.mu_y);
      if (mp != own && mm != own) return;
      const int ex = along_x ? e : x, ey = along_x ? y : e, vx = along_x ? v : x, vy = along_x ? y : v;
      const T e0 = ld_phi(st, g, ex, ey, 0), e1 = ld_phi(st, g, ex, ey, 1);
      const T v0 = ld_phi(st, g, vx, vy, 0), v1 = ld_phi(st, g, vx, vy, 1);
      const T ge = cell_ldc(m, e0, e1, lmu_in[(int64_t)ex * g.pitch + ey]) * m.dt;
      const T ue = st[2 * g.plane + (int64_t)ex * g.pitch + ey], uv = ld_mu(st, g, vx, vy);
      const T Ds2 = (k0 * v0 + k1 * v1) + (k0 * e0 + k1 * e1);
      if (low) gather((T)1, (T)0, ge, uv, ue, Ds2, (T)0, along_x ? 0 : 1, mp == own, mm == own);
      else gather((T)-1, ge, (T)0, ue, uv, Ds2, (T)0, along_x ? 0 : 1, mp == own, mm == own);
    };
    if (x <= 2 || x >= g.mx - 3) {
      ghost(true, true);
      ghost(true, false);
    }
    if (y <= 2 || y >= g.my - 3) {
      ghost(false, true);
      ghost(false, false);
    }
    lam_out[o] = lph[0] + sD * k0;
    lam_out[g.plane + o] = lph[1] + sD * k1;
    lam_out[2 * g.plane + o] = lmu + sM;
  }
  block_add(dl, part + blockIdx.x);
}

// Scatter of one adjoint contribution; a zero one is skipped.
template <typename T>
__device__ __forceinline__ void add_nz(T* p, T v) {
  if (v != (T)0) atomicAdd(p, v);
}

// 2. reverse of the antitrapping currents: a thread per face of a listed ring cell (k as in
// cell_face).  A face between two listed cells belongs to its lower one; one whose lower cell is flat
// to its upper one.  Faces between two flat cells carry no current and no derivative.
// Bound by latency (a few thousand threads with one dependent chain of square roots and divisions).
template <typename T, bool POW2>
__global__ void __launch_bounds__(128) k_rev_jat(const __grid_constant__ AM<T, POW2> m, Geo g, const T* st, const T* ring,
                                                 const T* lam_in, T* lam_out, T* ldphi, const int* list,
                                                 const int* cnt, double* part) {
  begin_dependent();
  double dl = 0.0;
  const int64_t thread = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, threads = gridDim.x * (int64_t)blockDim.x;
  for (ListWalk q(*cnt, 4, thread, threads); q.more(); q.next()) {
    const int o = list[q.at >> 2], k = (int)(q.at & 3), dir = k >> 1;
    int x = o / g.rpitch - 1, y = o % g.rpitch - 1;  // the listed cell, then the face's lower cell
    if (k & 1) {
      if (dir == 0) x--;
      else y--;
    }
    const bool valid = dir == 0 ? (x >= -1 && x < g.mx && y >= 0 && y < g.my) : (y >= -1 && y < g.my && x >= 0 && x < g.mx);
    if (!valid) continue;
    if (k & 1) {
      T P[3][3][2];
      load_P(st, g, x, y, P);
      if (!flat_P(P)) continue;
    }
    const int xn = dir == 0 ? x + 1 : x, yn = dir == 0 ? y : y + 1;
    const T h = dir == 0 ? m.dx : m.dy;
    Face<T> f;
    for (int a = 0; a < 2; a++) {
      f.pc[a] = ld_phi(st, g, x, y, a);
      f.pn[a] = ld_phi(st, g, xn, yn, a);
      if (dir == 0) {
        f.tc[a] = m.qt(ld_phi(st, g, x, y + 1, a) - ld_phi(st, g, x, y - 1, a));
        f.tn[a] = m.qt(ld_phi(st, g, xn, y + 1, a) - ld_phi(st, g, xn, y - 1, a));
      } else {
        f.tc[a] = (T)0.5 * (m.qx(ld_phi(st, g, x + 1, y, a) - f.pc[a]) + m.qx(f.pc[a] - ld_phi(st, g, x - 1, y, a)));
        f.tn[a] = (T)0.5 * (m.qx(ld_phi(st, g, x + 1, yn, a) - f.pn[a]) + m.qx(f.pn[a] - ld_phi(st, g, x - 1, yn, a)));
      }
    }
    T lc = (T)0, ln = (T)0;  // the two cells' divjat adjoints
    if (x >= 0 && y >= 0) lc = -cell_ldc(m, f.pc[0], f.pc[1], lam_in[2 * g.plane + (int64_t)x * g.pitch + y]);
    if (xn < g.mx && yn < g.my) ln = -cell_ldc(m, f.pn[0], f.pn[1], lam_in[2 * g.plane + (int64_t)xn * g.pitch + yn]);
    const T lJ = m.qd(dir, (lc - ln) * m.jscale);
    if (lJ == (T)0) continue;
    f.muc = ld_mu(st, g, x, y);
    f.mun = ld_mu(st, g, xn, yn);
    f.dpc = ring[ix_ring(g, x, y, 0)];
    f.dpn = ring[ix_ring(g, xn, yn, 0)];
    f.h = h;
    f.ih = dir == 0 ? m.ix : m.iy;
    f.skip = dir == 1 && (y + 3 == g.my - 2);
    FaceAdj<T> L = {};
    T lp[NPARAM] = {(T)0, (T)0, (T)0, (T)0};
    jface_rev(m, f, lJ, L, lp);
    dl += (double)lp[P_DLIQ];
    for (int a = 0; a < 2; a++) {
      add_nz(lam_out + ix_phi(g, x, y, a), L.pc[a]);
      add_nz(lam_out + ix_phi(g, xn, yn, a), L.pn[a]);
      if (dir == 0) {
        const T hc = m.qt(L.tc[a]), hn = m.qt(L.tn[a]);
        add_nz(lam_out + ix_phi(g, x, y + 1, a), hc);
        add_nz(lam_out + ix_phi(g, x, y - 1, a), -hc);
        add_nz(lam_out + ix_phi(g, xn, y + 1, a), hn);
        add_nz(lam_out + ix_phi(g, xn, y - 1, a), -hn);
      } else {
        const T hc = m.qx((T)0.5 * L.tc[a]), hn = m.qx((T)0.5 * L.tn[a]);
        add_nz(lam_out + ix_phi(g, x + 1, y, a), hc);
        add_nz(lam_out + ix_phi(g, x - 1, y, a), -hc);
        add_nz(lam_out + ix_phi(g, x + 1, yn, a), hn);
        add_nz(lam_out + ix_phi(g, x - 1, yn, a), -hn);
      }
    }
    add_nz(lam_out + ix_mu(g, x, y), L.muc);
    add_nz(lam_out + ix_mu(g, xn, yn), L.mun);
    add_nz(ldphi + ix_ring(g, x, y, 0), L.dpc);
    add_nz(ldphi + ix_ring(g, xn, yn, 0), L.dpn);
  }
  block_add(dl, part + blockIdx.x);
}

// 3. reverse of Delta-phi (the pieces of dphi_rev, gp_adjoint_cell.cuh) on the listed ring cells, eight lanes
// per cell: lane a * 4 + k reverses face k of phase a's gradient-energy term, the terms at the cell's
// centre and the projection are evaluated by all eight, and lanes 0 and 1 of each phase scatter the
// centre's contributions with their faces'.  One thread per cell is a chain of twenty a_c(q)
// evaluations with their reverses on a few thousand threads, far too few to hide it.
template <typename T, bool POW2>
__global__ void __launch_bounds__(128) k_rev_dphi(const __grid_constant__ AM<T, POW2> m, Geo g, const T* st, const T* ldphi,
                                                  T* lam_out, const int* list, const int* cnt, double* part) {
  begin_dependent();
  constexpr unsigned ALL = 0xffffffffu;
  double acc[3] = {0.0, 0.0, 0.0};  // mobility, delta, gamma
  const int lane = threadIdx.x & 31, sub = lane & 7, a = sub >> 2, k = sub & 3;
  const int n = *cnt, warps = (gridDim.x * blockDim.x) >> 5, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (ListWalk four(n, 1, 4 * warp, 4 * warps); four.more(); four.next()) {  // four cells a warp
    const int64_t q = four.at + (lane >> 3);
    const int o = list[q < n ? q : n - 1], x = o / g.rpitch - 1, y = o % g.rpitch - 1;
    const T ldp[2] = {q < n ? ldphi[o] : (T)0, q < n ? ldphi[o + g.rplane] : (T)0};
    bool on = ldp[0] != (T)0 || ldp[1] != (T)0;
    if (!__any_sync(ALL, on)) continue;
    T P[3][3][2];
    load_P(st, g, x, y, P);
    const T mu = ld_mu(st, g, x, y);
    DCell<T> c;
    dphi_cell(m, P, c);
    on = on && (c.act[0] || c.act[1]);  // no active phase: Delta-phi is 0 whatever the inputs
    DLane<T> L;
    dphi_lane(m, P, c, a, k, L);
    T sum4 = dphi_face(m, L, a, k);
    sum4 += __shfl_xor_sync(ALL, sum4, 1);
    sum4 += __shfl_xor_sync(ALL, sum4, 2);
    DTerm<T> t;
    dphi_term(m, c, L, mu, a, sum4, t);
    const T lam_o = __shfl_xor_sync(ALL, t.lam, 4);
    T lph[2], dmob;
    const T la = dphi_mean_rev(m, c, a ? lam_o : t.lam, a ? t.lam : lam_o, ldp, a, lph, dmob);
    const bool lane_on = on && L.act_a;  // an inactive phase's operands may have overflowed
    DAdj<T> o8;
    dphi_lane_rev(m, L, t, mu, a, k, sum4, lane_on ? la : (T)0, o8);
    T lmu = lane_on ? o8.lmu : (T)0;
    acc[1] += lane_on ? (double)o8.ldab : 0.0;
    acc[2] += lane_on ? (double)o8.lgam : 0.0;
    lmu += __shfl_xor_sync(ALL, lmu, 4);
    if (on && sub == 0) {
      acc[0] += (double)dmob;
      add_nz(lam_out + ix_mu(g, x, y), lmu);
    }
    // The partner lane (the other phase) holds the same cells' other half, exchanged so that a lane has one
    // phase's values; the projection's own adjoints go with the first lane's centre.
    T v[2][3];
#pragma unroll
    for (int nn = 0; nn < 2; nn++)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        T mine = lane_on ? o8.v[0][nn][i] : (T)0, other = lane_on ? o8.v[1][nn][i] : (T)0;
        if (nn == 0 && i == 1 && sub == 0) {
          mine += lph[0];
          other += lph[1];
        }
        v[nn][i] = mine + __shfl_xor_sync(ALL, other, 4);
      }
    // The four faces' sums, so that each of the nine cells takes one addition (24 before: each a rounding at
    // the scale of the adjoint, and an atomic).  The x faces' lanes hold rows (k = 0: 1 and 2, k = 1: 0
    // and 1), the y faces' columns; the middle row and column go to the even lanes, then each cell's row part
    // meets its column part.
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const T middle = __shfl_xor_sync(ALL, v[1][i], 1);
      if (!(k & 1)) v[0][i] += middle;
    }
    const T *const lo = v[0], *const up = v[1];
    const T r0 = __shfl_xor_sync(ALL, k == 0 ? up[1] : k == 1 ? lo[0] : lo[1], 2);
    const T r1 = __shfl_xor_sync(ALL, k == 0 ? up[2] : up[1], 2);
    const T r2 = __shfl_xor_sync(ALL, k == 0 ? up[0] : k == 1 ? lo[2] : k == 2 ? lo[0] : lo[1], 3);
    if (!on) continue;
    auto add = [&](int dx, int dy, T w) { add_nz(lam_out + ix_phi(g, x + dx, y + dy, a), w); };
    if (k == 0) {
      add(0, 0, lo[1] + r0);
      add(0, 1, lo[2] + r1);
      add(0, -1, lo[0] + r2);
    } else if (k == 1) {
      add(-1, 0, lo[1] + r2);
    } else if (k == 2) {
      add(1, 0, lo[2] + r0);
      add(1, 1, up[2] + r1);
      add(-1, 1, up[0] + r2);
    } else {
      add(1, -1, lo[2] + r2);
      add(-1, -1, lo[0] + r0);
    }
  }
#pragma unroll
  for (int p = 0; p < 3; p++) block_add(acc[p], part + 3 * blockIdx.x + p);
}

// The parameter gradients from the blocks' sums: thread block p, a fixed order.
__global__ void __launch_bounds__(256) k_grad(const double* __restrict__ cell, int ncell,
                                              const double* __restrict__ jat, int njat,
                                              const double* __restrict__ dphi, int ndphi, double* __restrict__ grad) {
  const int p = blockIdx.x;
  double v = 0.0;
  if (p == P_DLIQ) {
    for (int i = threadIdx.x; i < ncell; i += blockDim.x) v += cell[i];
    for (int i = threadIdx.x; i < njat; i += blockDim.x) v += jat[i];
  } else {
    for (int i = threadIdx.x; i < ndphi; i += blockDim.x) v += dphi[3 * i + p];
  }
  if (threadIdx.x == 0) grad[p] = 0.0;
  block_add(v, grad + p);
}

// Values start .. start + n - 1 of dense FP64 host planes, staged on the device, <-> the planes at st.
template <typename T>
__global__ void __launch_bounds__(256) k_fields(T* __restrict__ st, double* __restrict__ stage, Geo g, int64_t start,
                                                int64_t n, int up) {
  const int64_t cells = (int64_t)g.mx * g.my;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = (start + i) / cells, r = (start + i) % cells;
    const int64_t o = p * g.plane + (r / g.my) * g.pitch + r % g.my;
    if (up) st[o] = (T)stage[i];
    else stage[i] = (double)st[o];
  }
}

// ------------------------------------------------------------------ host side

template <typename T, bool POW2>
AM<T, POW2> make_am(const gp_model& g) {
  AM<T, POW2> m;
  m.dx = (T)g.dx;
  m.dy = (T)g.dy;
  m.dt = (T)g.dt;
  m.eps = (T)g.epsilon;
  m.inv_eps = (T)g.inv_eps;
  m.mob = (T)(1.0 / g.tau_ab[0][1]);
  m.tau_ratio = (T)(g.tau / g.tau_ab[0][1]);
  m.gam = (T)g.Gamma[0][1];
  m.dab = g.anisotropy ? (T)g.dab[0][1] : (T)0;
  m.wobs = (T)g.w_obstacle;
  m.jscale = (T)(g.obstacle ? g.jat_obst : g.jat_well);
  m.swell = (T)g.s_well;
  for (int a = 0; a < 2; a++)
    for (int i = 0; i < 2; i++)
      for (int j = 0; j < 2; j++) {
        m.R[a][i][j] = g.anisotropy ? (T)g.R[a][1 - a][i][j] : (T)(i == j);
        m.Ri[a][i][j] = g.anisotropy ? (T)g.Rinv[a][1 - a][i][j] : (T)(i == j);
      }
  for (int a = 0; a < 2; a++) {
    m.cmu[a] = (T)g.cmu[a][0][0];
    m.A[a] = (T)g.A[a][0][0];
    m.B[a] = (T)g.B[a][0];
    m.C[a] = (T)g.C[a];
    m.Beff[a] = (T)g.Beff[a][0];
  }
  m.Ds = (T)g.Diff[0][0][0];
  m.Dl = (T)g.Diff[1][0][0];
  m.obstacle = g.obstacle ? 1 : 0;
  m.skip_row = (int)g.mesh_y - 5;
  m.ix = (T)1 / m.dx;
  m.iy = (T)1 / m.dy;
  m.it = (T)1 / ((T)2 * m.dy);
  return m;
}

struct AdjBase {
  virtual ~AdjBase() {}
  virtual int forward(const double* phi0, const double* mu0, int64_t nsteps, int64_t every, double* phi_out,
                      double* mu_out) = 0;
  virtual int backward(const double* lphi, const double* lmu, double* grad, double* lphi0, double* lmu0) = 0;
  int64_t stored = 0;
};

#define ADJ_CUDA(call)                                                                  \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      gp_set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_));  \
      return GP_E_CUDA;                                                                 \
    }                                                                                   \
  } while (0)

template <typename T>
struct Adj : AdjBase {
  gp_model gm;
  // the spacings' quotients as products where dx and dy are powers of two (a template switch: the list
  // kernels wait for their instructions, and a division is ten times a product's)
  AM<T, true> mp;
  AM<T, false> md;
  bool pow2 = false;
  Geo g;
  cudaStream_t s = nullptr;
  T *cur = nullptr, *nxt = nullptr;
  // one allocation for what a run keeps (reserve): the checkpoints, a segment's states and their slots below
  char* arena = nullptr;
  int64_t arena_bytes = 0, refused = 0;  // refused: an allocation of that size failed
  T *ckpt = nullptr, *seg = nullptr;
  // Delta-phi, list of the cells that are not flat and its length: of every state of a segment
  // (slots == every), or of one state at a time, recomputed before its reverse, where that
  // does not fit (slots == 1)
  T* ring = nullptr;
  int *list = nullptr, *cnt = nullptr;
  int64_t slots = 0;
  T *lam[2] = {nullptr, nullptr}, *ldphi = nullptr;
  double *part = nullptr, *dgrad = nullptr, *stage = nullptr;
  int ntile = 0, nlist = 0;  // blocks of the dense kernels and of the list kernels
  int64_t nsteps = 0, every = 0, nck = 0;
  bool have = false;

  int64_t state() const { return 3 * g.plane; }

  ~Adj() {
    if (s) cudaStreamSynchronize(s);
    cudaFree(arena);
    cudaFree(cur);
    cudaFree(nxt);
    cudaFree(lam[0]);
    cudaFree(lam[1]);
    cudaFree(ldphi);
    cudaFree(part);
    cudaFree(dgrad);
    cudaFree(stage);
    if (s) cudaStreamDestroy(s);
  }

  int init(const gp_model& model) {
    gm = model;
    mp = make_am<T, true>(model);
    md = make_am<T, false>(model);
    g.mx = (int)model.mesh_x;
    g.my = (int)model.mesh_y;
    g.pitch = (int)gp_round_up(g.my, 32);
    g.plane = (int64_t)g.pitch * g.mx;
    g.rpitch = (int)gp_round_up(g.my + 2, 32);
    g.rplane = (int64_t)g.rpitch * (g.mx + 2);
    g.bc = gp_bc_of(model);
    if (g.rplane > INT32_MAX) {
      gp_set_error("adjoint: %d x %d cells do not fit", g.mx, g.my);
      return GP_E_NOMEM;
    }
    int ex, ey;
    pow2 = frexp(model.dx, &ex) == 0.5 && frexp(model.dy, &ey) == 0.5 && abs(ex) < 60 && abs(ey) < 60;
    int dev = 0, sms = 0;
    ADJ_CUDA(cudaGetDevice(&dev));
    ADJ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    ntile = ((g.mx + TX - 1) / TX) * ((g.my + TY - 1) / TY);
    nlist = 4 * sms;
    ADJ_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    ADJ_CUDA(cudaMalloc(&cur, sizeof(T) * state()));
    ADJ_CUDA(cudaMalloc(&nxt, sizeof(T) * state()));
    ADJ_CUDA(cudaMalloc(&lam[0], sizeof(T) * state()));
    ADJ_CUDA(cudaMalloc(&lam[1], sizeof(T) * state()));
    ADJ_CUDA(cudaMalloc(&ldphi, sizeof(T) * 2 * g.rplane));
    ADJ_CUDA(cudaMalloc(&part, sizeof(double) * ((int64_t)ntile + 4 * nlist)));
    ADJ_CUDA(cudaMalloc(&dgrad, sizeof(double) * NPARAM));
    ADJ_CUDA(cudaMemsetAsync(cur, 0, sizeof(T) * state(), s));
    ADJ_CUDA(cudaMemsetAsync(nxt, 0, sizeof(T) * state(), s));
    return GP_OK;
  }

  cudaError_t step(const T* in, T* out, T* r = nullptr, int* l = nullptr, int* c = nullptr) {
    return pow2 ? gp_launch_dependent(k_fwd<T, true>, ntile, NT, 0, s, mp, g, in, out, r, l, c)
                : gp_launch_dependent(k_fwd<T, false>, ntile, NT, 0, s, md, g, in, out, r, l, c);
  }

  // lin = adjoint of the state after x, lout = adjoint of x; r, l, c: x's Delta-phi, list and its length
  cudaError_t rev_step(const T* x, const T* r, const int* l, const int* c, const T* lin, T* lout) {
    return pow2 ? rev_step(mp, x, r, l, c, lin, lout) : rev_step(md, x, r, l, c, lin, lout);
  }
  template <bool POW2>
  cudaError_t rev_step(const AM<T, POW2>& m, const T* x, const T* r, const int* l, const int* c, const T* lin, T* lout) {
    cudaError_t e = gp_launch_dependent(k_rev_cell<T, POW2>, ntile, NT, 0, s, m, g, x, r, lin, lout, ldphi, part);
    if (e == cudaSuccess)
      e = gp_launch_dependent(k_rev_jat<T, POW2>, nlist, 128, 0, s, m, g, x, r, lin, lout, ldphi, l, c, part + ntile);
    if (e == cudaSuccess)
      e = gp_launch_dependent(k_rev_dphi<T, POW2>, nlist, 128, 0, s, m, g, x, ldphi, lout, l, c, part + ntile + nlist);
    return e;
  }

  // Host [planes][mx][my] doubles <-> device [planes][mx][pitch] T, converted on the device through a
  // staging buffer of at most kStage doubles (the conversion of a 512^2 state on a host core took
  // longer than its 100 steps).  An upload without a host array is zeros.
  static constexpr int64_t kStage = 4 << 20;
  int move(T* planes, int nplanes, double* host, bool up) {
    const int64_t all = (int64_t)nplanes * g.mx * g.my;
    if (!host) {
      if (up) ADJ_CUDA(cudaMemsetAsync(planes, 0, sizeof(T) * nplanes * g.plane, s));
      return GP_OK;
    }
    const int64_t room = 3ll * g.mx * g.my < kStage ? 3ll * g.mx * g.my : kStage;
    if (!stage) ADJ_CUDA(cudaMalloc(&stage, sizeof(double) * room));
    for (int64_t at = 0; at < all; at += room) {
      const int64_t n = all - at < room ? all - at : room;
      if (up) ADJ_CUDA(cudaMemcpyAsync(stage, host + at, sizeof(double) * n, cudaMemcpyHostToDevice, s));
      k_fields<T><<<592, 256, 0, s>>>(planes, stage, g, at, n, up ? 1 : 0);
      ADJ_CUDA(cudaGetLastError());
      if (!up) ADJ_CUDA(cudaMemcpyAsync(host + at, stage, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    }
    return GP_OK;
  }
  int upload(T* dst, const double* phi, const double* mu) {
    int rc = move(dst, 2, const_cast<double*>(phi), true);
    return rc == GP_OK ? move(dst + 2 * g.plane, 1, const_cast<double*>(mu), true) : rc;
  }
  int download(T* src, double* phi, double* mu) {
    int rc = move(src, 2, phi, false);
    if (rc == GP_OK) rc = move(src + 2 * g.plane, 1, mu, false);
    if (rc == GP_OK) ADJ_CUDA(cudaStreamSynchronize(s));
    return rc;
  }

  // Bytes of nc checkpoints, ev segment states and n slots, and their places in the arena.
  struct Layout {
    int64_t states, rings, lists, all;
  };
  Layout layout(int64_t nc, int64_t ev, int64_t n) const {
    Layout y;
    y.states = sizeof(T) * state() * (nc + ev);
    y.rings = sizeof(T) * 2 * g.rplane * n;
    y.lists = sizeof(int) * g.rplane * n;
    y.all = y.states + y.rings + y.lists + sizeof(int) * n;
    return y;
  }

  // Room for nc checkpoints, ev segment states and their slots.  A slot of its own for every state (about as
  // much again as the states) saves recomputing its Delta-phi; it is taken where that leaves half of
  // the device's free memory to others, else one slot serves all.  The arena is kept for later runs, but not
  // at more than four times (and 64 MB) what a run needs.
  bool reserve(int64_t nc, int64_t ev) {
    int64_t n = ev;
    Layout y = layout(nc, ev, n);
    if (arena_bytes < y.all && ev > 1) {
      size_t room = 0, total = 0;
      if (cudaMemGetInfo(&room, &total) != cudaSuccess) cudaGetLastError();
      if (y.all > ((int64_t)room + arena_bytes) / 2 || (refused && y.all >= refused)) y = layout(nc, ev, n = 1);
    }
    for (;; y = layout(nc, ev, n = 1)) {
      if (arena_bytes < y.all || arena_bytes > 4 * y.all + (64 << 20)) {
        cudaFree(arena);
        arena = nullptr;
        arena_bytes = 0;
        if (cudaMalloc(&arena, y.all) == cudaSuccess) arena_bytes = y.all;
        else cudaGetLastError();
      }
      if (arena_bytes >= y.all) break;
      if (n == 1) return false;
      refused = y.all;  // not tried again by this object
    }
    ckpt = reinterpret_cast<T*>(arena);
    seg = ckpt + state() * nc;
    ring = reinterpret_cast<T*>(arena + y.states);
    list = reinterpret_cast<int*>(arena + y.states + y.rings);
    cnt = reinterpret_cast<int*>(arena + y.states + y.rings + y.lists);
    slots = n;
    return true;
  }

  int forward(const double* phi0, const double* mu0, int64_t n, int64_t ev, double* phi_out,
              double* mu_out) override {
    if (n < 1 || !phi0 || !mu0) return GP_E_ARG;
    if (ev <= 0) ev = (int64_t)ceil(sqrt((double)n));
    if (ev > n) ev = n;
    const int64_t nc = (n + ev - 1) / ev;
    have = false;
    ADJ_CUDA(cudaStreamSynchronize(s));  // nothing queued reads the arena, which may be replaced
    if (!reserve(nc, ev)) {
      gp_set_error("adjoint: %lld checkpoints + %lld segment states do not fit", (long long)nc, (long long)ev);
      return GP_E_NOMEM;
    }
    nsteps = n;
    every = ev;
    nck = nc;
    stored = nc + ev;
    int rc = upload(cur, phi0, mu0);
    if (rc != GP_OK) return rc;
    for (int64_t i = 0; i < n; i++) {
      if (i % ev == 0)
        ADJ_CUDA(cudaMemcpyAsync(ckpt + (i / ev) * state(), cur, sizeof(T) * state(), cudaMemcpyDeviceToDevice, s));
      ADJ_CUDA(step(cur, nxt));
      T* t = cur;
      cur = nxt;
      nxt = t;
    }
    have = true;
    return download(cur, phi_out, mu_out);
  }

  int backward(const double* lphi, const double* lmu, double* grad, double* lphi0, double* lmu0) override {
    if (!have) {
      gp_set_error("adjoint: backward before forward");
      return GP_E_ARG;
    }
    if (!grad) return GP_E_ARG;
    int rc = upload(lam[0], lphi, lmu);
    if (rc != GP_OK) return rc;
    ADJ_CUDA(cudaMemsetAsync(part, 0, sizeof(double) * ((int64_t)ntile + 4 * nlist), s));
    const bool all = slots >= every;  // every state of a segment has its slot
    int li = 0;
    for (int64_t k = nck - 1; k >= 0; k--) {
      const int64_t start = k * every, len = (nsteps - start < every) ? nsteps - start : every;
      const T* const first = ckpt + k * state();
      auto at = [&](int64_t i) { return i ? seg + i * state() : first; };
      if (all) ADJ_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * len, s));
      for (int64_t i = 1; i < len; i++)
        ADJ_CUDA(all ? step(at(i - 1), seg + i * state(), ring + (i - 1) * 2 * g.rplane, list + (i - 1) * g.rplane, cnt + (i - 1))
                     : step(at(i - 1), seg + i * state()));
      for (int64_t i = len - 1; i >= 0; i--) {
        const int64_t q = all ? i : 0;
        T* const r = ring + q * 2 * g.rplane;
        int* const l = list + q * g.rplane;
        if (!all) ADJ_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int), s));
        if (!all || i == len - 1) ADJ_CUDA(step(at(i), nullptr, r, l, cnt + q));
        ADJ_CUDA(rev_step(at(i), r, l, cnt + q, lam[li], lam[li ^ 1]));
        li ^= 1;
      }
    }
    k_grad<<<NPARAM, 256, 0, s>>>(part, ntile, part + ntile, nlist, part + ntile + nlist, nlist, dgrad);
    ADJ_CUDA(cudaGetLastError());
    ADJ_CUDA(cudaMemcpyAsync(grad, dgrad, sizeof(double) * NPARAM, cudaMemcpyDeviceToHost, s));
    ADJ_CUDA(cudaStreamSynchronize(s));
    if (lphi0 || lmu0) return download(lam[li], lphi0, lmu0);
    return GP_OK;
  }
};

}  // namespace

struct gp_adj {
  AdjBase* impl;
};

extern "C" int gp_adj_create(const gp_model* m, int precision, gp_adj** out) {
  if (!m || !out) return GP_E_ARG;
  *out = nullptr;
  if (m->N != 2 || m->K1 != 1) {
    gp_set_error("adjoint: binary alloys only (N = 2, K-1 = 1), got N = %d, K-1 = %d", m->N, m->K1);
    return GP_E_UNSUPPORTED;
  }
  if (m->mesh_x < 4 || m->mesh_y < 4) return GP_E_ARG;
  if (m->nonisothermal) {
    gp_set_error("adjoint: isothermal models only");
    return GP_E_UNSUPPORTED;
  }
  gp_adj* a = new gp_adj();
  int rc;
  if (precision == GP_FP32) {
    Adj<float>* p = new Adj<float>();
    a->impl = p;
    rc = p->init(*m);
  } else {
    Adj<double>* p = new Adj<double>();
    a->impl = p;
    rc = p->init(*m);
  }
  if (rc != GP_OK) {
    delete a->impl;
    delete a;
    return rc;
  }
  *out = a;
  return GP_OK;
}

extern "C" int gp_adj_forward(gp_adj* a, const double* phi0, const double* mu0, int64_t nsteps,
                              int64_t checkpoint_every, double* phi_out, double* mu_out) {
  if (!a) return GP_E_ARG;
  return a->impl->forward(phi0, mu0, nsteps, checkpoint_every, phi_out, mu_out);
}

extern "C" int gp_adj_backward(gp_adj* a, const double* lam_phi, const double* lam_mu, double* grad,
                               double* lam_phi0, double* lam_mu0) {
  if (!a) return GP_E_ARG;
  return a->impl->backward(lam_phi, lam_mu, grad, lam_phi0, lam_mu0);
}

extern "C" int gp_adj_stored_states(const gp_adj* a, int64_t* states) {
  if (!a || !states) return GP_E_ARG;
  *states = a->impl->stored;
  return GP_OK;
}

extern "C" int gp_adj_destroy(gp_adj* a) {
  if (!a) return GP_OK;
  delete a->impl;
  delete a;
  return GP_OK;
}
