// tile2d.h - 2-D modes: several time steps per launch (tile2d.cuh).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "params.h"

namespace fdtdb {

constexpr int kTileSteps = 7;   // steps per launch at most: the halo of a tile

// One component of a 2-D mode.  The kept axes are u (first) and v (second,
// contiguous); a cell's index is u nv + v.
struct TileComp
{
  int nmat, m[4][2];           // material stencil
  const void *mat;             // double (FP64) or float; null: 1
  const void *in, *aux_in;     // current level: field and PML auxiliary (null without PML)
  void *out, *aux_out;         // level after the steps
  const void *tab[6];          // PML tables: PlainTabs (FP64) or FastHalf order
  int ilo[2], ihi[2];          // FP32: sigma = 0 range
  int source;                  // a point source drives it
  int nterms;
  TermDev term[kMaxTerms];     // lo, hi, aux of the axes u, v in [0], [1]
};

// Shape of a 2-D mode: te: two E components in the plane and one H across it
// (else one E across, two H in the plane); flip: the kept axes and the
// dropped one in the cyclic order u, w, v (y dropped); hc: H_CENTERED.
struct TileForm
{
  bool te, flip, hc;
};

struct Tile2D
{
  TileForm form;
  int nu, nv;
  int use_pml;
  int steps;                   // 1 .. kTileSteps, odd in FP64
  TileComp comp[3];            // E components (u, then v), then H
  double mm[2];                // FP64: eps0, mu0
  double dt, dx;
  float courant;               // FP32
  float scale[2];              // FP32: field units of E, H (1, eta0)
  // point source cell; source table: src_row values per step, the incident
  // grid's source first, then the point source on E and on H
  int pu, pv;
  const double *src;
  int src_row;
  // TF/SF: the 1-D grid (current and next level) and the incident distance
  int use_tfsf;
  const double *e_in, *h_in;
  double *e_out, *h_out;
  int inc_len, inc_cells;      // length; cells that may differ from 0 after the steps
  double mod_e, mod_h;
  double k[2], zero[2], proj[6], pos[6][2];
  int *err;
};

// Advances every cell by p.steps time steps (t > 0) in one launch: fields,
// auxiliaries and the incident grid from their current to their next level.
int launch_tile2d_fp64 (const Tile2D &p, int sm_count, cudaStream_t s);
int launch_tile2d_fast (const Tile2D &p, bool fp16, int sm_count, cudaStream_t s);

}  // namespace fdtdb
