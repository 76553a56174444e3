// gp_tiles.cuh -- purity words of a grid's tiles: what lets a step skip the phase-field arithmetic of
// tiles far from every interface (FP32 form: lean kernels; plain form: the bulk path of its tile kernel).
//
// Far from every interface a cell's phi is the one-hot field of one phase and its update is diffusion
// of mu inside that phase.  Each step writes, per tile, a purity word describing its output: five
// 4-bit fields, each 1 + b when every in-grid cell of that part of the tile holds the one-hot field of
// phase b (exactly 1 and +0), else 0.  The parts: the whole tile, its first and last two rows (x) and
// its first and last two columns (y).
#pragma once

#include "gp_common.cuh"

enum { PF_CORE = 0, PF_XLO = 4, PF_XHI = 8, PF_YLO = 12, PF_YHI = 16 };
__host__ __device__ __forceinline__ int pf(uint32_t w, int f) { return (int)((w >> f) & 15u); }
__host__ __device__ __forceinline__ uint32_t pf_all(int c) { return (uint32_t)c * 0x11111u; }

// Static facts of tile t used by lean_phase, one word: tiles along y (the
// index stride of the x-neighbours), which of the four neighbours exist, and
// whether the tile is never lean (its two-cell ring leaves the grid where it
// is not a trusted mirror: a periodic wrap, or fewer than 3 cells on that axis).
// TG_REJECT2: the tile never takes the two-step lean update, because its two-cell
// ring leaves the grid across a periodic boundary of phi or mu (the ring's purity
// and the partner cells of the intermediate step are not known there).
enum : uint32_t { TG_NY = 0xFFFFFFu, TG_XM = 1u << 24, TG_XP = 1u << 25, TG_YM = 1u << 26, TG_YP = 1u << 27,
                  TG_REJECT = 1u << 28, TG_REJECT2 = 1u << 29 };

// k: the tile's index within its grid (tiles along y fastest).
inline uint32_t tile_geo(int mx, int my, const gp_bc& bc, int k, int TX, int TY) {
  const int nx = (mx + TX - 1) / TX, ny = (my + TY - 1) / TY, tx = k / ny, ty = k % ny;
  const int ex = mx - tx * TX < TX ? mx - tx * TX : TX, ey = my - ty * TY < TY ? my - ty * TY : TY;
  const bool xm = tx > 0, xp = tx + 1 < nx, ym = ty > 0, yp = ty + 1 < ny;
  const bool reject = ((!xm || !xp) && !(bc.phi_x == GP_BC_NEUMANN && ex >= 3)) ||
                      ((!ym || !yp) && !(bc.phi_y == GP_BC_NEUMANN && ey >= 3));
  const int x0 = tx * TX, y0 = ty * TY;
  const bool cross_x = x0 - 2 < 0 || x0 + TX + 2 > mx, cross_y = y0 - 2 < 0 || y0 + TY + 2 > my;
  const bool reject2 = (cross_x && (bc.phi_x != GP_BC_NEUMANN || bc.mu_x != GP_BC_NEUMANN)) ||
                       (cross_y && (bc.phi_y != GP_BC_NEUMANN || bc.mu_y != GP_BC_NEUMANN));
  return (uint32_t)ny | (xm ? TG_XM : 0u) | (xp ? TG_XP : 0u) | (ym ? TG_YM : 0u) | (yp ? TG_YP : 0u) |
         (reject ? TG_REJECT : 0u) | (reject2 ? TG_REJECT2 : 0u);
}

// Phase b >= 0 when tile t may take the lean update: in the input, the tile
// and the two-cell ring the full update reads around it (tile +- 2, the phi
// region it stages) hold the one-hot field of phase b, known from the purity
// words of the tile and its eight neighbours.  Where the ring leaves the grid
// it is the Neumann mirror of the tile's own cells (rows 1, 2 and M-2, M-3:
// the tile needs 3 cells on that axis); a periodic wrap is not trusted.
// The full update of such a tile is its pure-phase path, so the lean update
// gives the same bits.  -1 otherwise.  The nine words are loaded at once (a
// missing neighbour reads the tile's own word, unused).
__host__ __device__ __forceinline__ int lean_phase(const uint32_t* __restrict__ F, uint32_t geo, int t) {
  if (geo & TG_REJECT) return -1;
  const int ny = (int)(geo & TG_NY);
  const bool xm = geo & TG_XM, xp = geo & TG_XP, ym = geo & TG_YM, yp = geo & TG_YP;
  const uint32_t w = F[t];
  const uint32_t wxm = F[xm ? t - ny : t], wxp = F[xp ? t + ny : t], wym = F[ym ? t - 1 : t],
                 wyp = F[yp ? t + 1 : t];
  const uint32_t wmm = F[xm && ym ? t - ny - 1 : t], wmp = F[xm && yp ? t - ny + 1 : t],
                 wpm = F[xp && ym ? t + ny - 1 : t], wpp = F[xp && yp ? t + ny + 1 : t];
  const int c = pf(w, PF_CORE);
  bool ok = c != 0;
  ok &= !xm || pf(wxm, PF_XHI) == c;
  ok &= !xp || pf(wxp, PF_XLO) == c;
  ok &= !ym || pf(wym, PF_YHI) == c;
  ok &= !yp || pf(wyp, PF_YLO) == c;
  ok &= !(xm && ym) || pf(wmm, PF_XHI) == c || pf(wmm, PF_YHI) == c;
  ok &= !(xm && yp) || pf(wmp, PF_XHI) == c || pf(wmp, PF_YLO) == c;
  ok &= !(xp && ym) || pf(wpm, PF_XLO) == c || pf(wpm, PF_YHI) == c;
  ok &= !(xp && yp) || pf(wpp, PF_XLO) == c || pf(wpp, PF_YLO) == c;
  return ok ? c - 1 : -1;
}
