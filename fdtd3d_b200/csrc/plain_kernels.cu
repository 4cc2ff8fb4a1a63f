// plain_kernels.cu - FP64 kernels compiled with --fmad=false.
//
// * plain_half_kernel: one half-step (all E or all H components) of the FP64
//   plain form, one thread per interior cell, curl -> Drude -> E-from-D fused
//   per cell.  Replaces the reference's per-component
//   calculateFieldStepIterationKernel, ...PMLMetamaterialsKernel and
//   ...PMLKernel launches plus their <<<1,1>>> shiftInTime kernels
//   (Source/Scheme/InternalScheme.inc.h:21-432); time levels rotate as kernel
//   arguments instead.
// * incident_e_kernel / incident_h_kernel: the 1-D auxiliary TF/SF grid
//   (InternalScheme.inc.h:3276-3357), FP64 for every form.
// * point_source_kernel: hard sinusoidal source (InternalScheme.inc.h:2818-2895).
// * fine_average_kernel: double material precision - one component's
//   material, averaged over the eight fine cells around it
//   (YeeGridLayout.h:866-1030, Approximation.cpp:34-54), once per upload.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "cell_walk.cuh"
#include "kernels.h"
#include "plain_cell.cuh"

namespace fdtdb {

template <bool DMP, bool CS>
__global__ void __launch_bounds__ (256) plain_half_kernel (PlainHalf p, int inc_len, int *err)
{
  // interior cells: 1 .. n - 2 on every axis a mode keeps, 0 on a dropped one
  const int ix = (p.g.drop & 1) ? 1 : p.g.n[0] - 2;
  const int iy = (p.g.drop & 2) ? 1 : p.g.n[1] - 2;
  const int iz = (p.g.drop & 4) ? 1 : p.g.n[2] - 2;
  const int64_t total = (int64_t) ix * iy * iz;
  for (int64_t tid = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; tid < total;
       tid += (int64_t) gridDim.x * blockDim.x)
  {
    const int z = (int) (tid % iz) + ((p.g.drop & 4) ? 0 : 1);
    const int64_t r = tid / iz;
    const int y = (int) (r % iy) + ((p.g.drop & 2) ? 0 : 1);
    const int x = (int) (r / iy) + ((p.g.drop & 1) ? 0 : 1);
#pragma unroll
    for (int ci = 0; ci < 3; ++ci)
    {
      if (p.comp[ci].exists)
        plain_component<DMP, CS> (p, ci, inc_len, err, x, y, z);
    }
  }
}

__global__ void incident_e_kernel (IncidentJob j)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < j.cells; i += gridDim.x * blockDim.x)
  {
    if (i == 0)
      j.now[0] = *j.src;
    else
      j.now[i] = j.old[i] + (j.other[i - 1] - j.other[i]) * j.modifier;
  }
}

__global__ void incident_h_kernel (IncidentJob j)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < j.cells; i += gridDim.x * blockDim.x)
    j.now[i] = j.old[i] + (j.other[i] - j.other[i + 1]) * j.modifier;
}

__global__ void incident_kernel (IncidentPair j)
{
  incident_pair (j, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__global__ void point_source_kernel (double *f, size_t index, const double *src, int src_index)
{
  if (threadIdx.x == 0 && blockIdx.x == 0)
    f[index] = src[src_index];
}

// The PML coefficient tables (PlainTabs): block y = component, block z =
// table pair; the expressions are plain_component's, so every value is the
// one the per-cell code computes at that coordinate.
struct PlainTabOut
{
  double *t[3][6];
};

__global__ void plain_tables_kernel (PlainHalf p, PlainTabOut o)
{
  const int ci = blockIdx.y, role = blockIdx.z;
  const CompDev &c = p.comp[ci];
  if (!c.exists)
    return;
  const double *const *sig = p.dmp ? p.sigc[ci] : p.sigma;
  const int axis = role == 0 ? c.sig_cacb : (role == 1 ? c.sig5 : c.sig4);
  const int n = p.g.n[axis];
  const double eps0 = kEps0Dev;
  const double dt = p.g.dt;
  const double dx = p.g.dx;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
  {
    bool inside = true;
    for (int j = 0; j < c.nmat; ++j)
      inside = inside && q + c.m[j][axis] >= 0 && q + c.m[j][axis] < n;
    if (!inside)
      continue;
    const double material = sigma_avg (c, sig[axis], axis, q, q, q);
    if (role == 0)
    {
      double dd = (2 * eps0 * 1.0 + material * dt);
      o.t[ci][0][q] = (2 * eps0 * 1.0 - material * dt) / dd;
      o.t[ci][1][q] = (2 * eps0 * dt / dx) / dd;
    }
    else if (role == 1)
    {
      double dd5 = (2 * eps0 * 1.0 + material * dt);
      o.t[ci][2][q] = (2 * eps0 * 1.0 - material * dt) / dd5;
      o.t[ci][3][q] = dd5;
    }
    else
    {
      o.t[ci][4][q] = (2 * eps0 * 1.0 + material * dt);
      o.t[ci][5][q] = (2 * eps0 * 1.0 - material * dt);
    }
  }
}

// One component of one half-step over every interior cell (the arithmetic
// of plain_component, parameters resolved before the cell loop).
template <bool PML, bool META, bool TFSF>
__global__ void __launch_bounds__ (256) plain_fast_kernel (const __grid_constant__ PlainHalf p,
                                                           const __grid_constant__ PlainTabs tb, int ncomp,
                                                           int inc_len, int *err)
{
  // block b updates component b % ncomp (of the existing ones) on cell block
  // b / ncomp: the blocks that read the same opposite-family cells run
  // together, so the later ones find them in L2
  int ci = 0;
  for (int k = 0, left = (int) (blockIdx.x % ncomp); k < 3; ++k)
    if (p.comp[k].exists && left-- == 0)
    {
      ci = k;
      break;
    }
  const int64_t cblock = blockIdx.x / ncomp, cgrid = gridDim.x / ncomp;
  const GeomDev &g = p.g;
  const CompDev &c = p.comp[ci];
  const int64_t sx = (int64_t) g.n[1] * g.n[2], sy = g.n[2];
  const int64_t d11 = c.d11[0] * sx + c.d11[1] * sy + c.d11[2];
  const int64_t d12 = c.d12[0] * sx + c.d12[1] * sy + c.d12[2];
  const int64_t d21 = c.d21[0] * sx + c.d21[1] * sy + c.d21[2];
  const int64_t d22 = c.d22[0] * sx + c.d22[1] * sy + c.d22[2];
  const int nmat = c.nmat;
  int64_t mo[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    mo[j] = c.m[j][0] * sx + c.m[j][1] * sy + c.m[j][2];
  const double *o1 = p.opp[c.opp1];
  const double *o2 = p.opp[c.opp2];
  const double *mat = p.dmp ? p.matc[ci] : p.mat;
  double *g0 = PML ? p.dd[ci][0] : p.f[ci][0];
  const double *g1 = PML ? p.dd[ci][1] : p.f[ci][1];
  const int ax_c = c.sig_cacb, ax5 = c.sig5, ax4 = c.sig4;
  const double *t_ca = tb.t[ci][0], *t_cb = tb.t[ci][1], *t_ca2 = tb.t[ci][2], *t_dd5 = tb.t[ci][3];
  const double *t_n4p = tb.t[ci][4], *t_n4m = tb.t[ci][5];
  const double dt = g.dt, dx = g.dx, mm = p.mat_modifier;
  double *f0 = p.f[ci][0];
  const double *f1 = p.f[ci][1];
  auto avg = [&] (const double *m, int64_t id) -> double {
    const double v0 = m[id + mo[0]];
    const double v1 = nmat > 1 ? m[id + mo[1]] : 0.0;
    const double v2 = nmat > 2 ? m[id + mo[2]] : 0.0;
    const double v3 = nmat > 3 ? m[id + mo[3]] : 0.0;
    return avg_points (nmat, v0, v1, v2, v3);
  };

  const int ix = (g.drop & 1) ? 1 : g.n[0] - 2;
  const int iy = (g.drop & 2) ? 1 : g.n[1] - 2;
  const int iz = (g.drop & 4) ? 1 : g.n[2] - 2;
  const int oz = (g.drop & 4) ? 0 : 1, oy = (g.drop & 2) ? 0 : 1, ox = (g.drop & 1) ? 0 : 1;
  for (CellWalk w (cblock * blockDim.x + threadIdx.x, cgrid * blockDim.x, ix, iy, iz); w.ok (); w.next ())
  {
    const int z = w.cz + oz, y = w.cy + oy, x = w.cx + ox;
    const int64_t id = x * sx + y * sy + z;
    const int pos[3] = {x, y, z};
    double val = g1[id];
    double ca, cb;
    if (PML)
    {
      const int q = ax_c == 0 ? x : (ax_c == 1 ? y : z);
      ca = t_ca[q];
      cb = t_cb[q];
    }
    else
    {
      double material = avg (mat, id);
      ca = 1.0;
      cb = dt / (material * mm * dx);
    }
    double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
    if (o1)
    {
      v0 = o1[id + d11];
      v1 = o1[id + d12];
    }
    if (o2)
    {
      v2 = o2[id + d21];
      v3 = o2[id + d22];
    }
    if (TFSF)
    {
      for (int t = 0; t < c.nterms; ++t)
      {
        const TermDev &tm = c.term[t];
        if (x >= tm.lo[0] && x < tm.hi[0] && y >= tm.lo[1] && y < tm.hi[1] && z >= tm.lo[2] && z < tm.hi[2])
        {
          double diff = incident_value (g, p.inc, inc_len, err, tm.inc_comp, x + tm.aux[0], y + tm.aux[1],
                                        z + tm.aux[2]);
          if (tm.negate < 0)
            diff *= -1.0;
          if (tm.slot == 0)
            v0 -= diff;
          else if (tm.slot == 1)
            v1 -= diff;
          else if (tm.slot == 2)
            v2 -= diff;
          else
            v3 -= diff;
        }
      }
    }
    double tmp = v1 - v0 - v3 + v2 - 0.0 * dx;
    double nv = val * ca + tmp * cb;
    g0[id] = nv;
    if (!PML)
      continue;
    if (META)
    {
      double cur = p.dd[ci][0][id], prev = p.dd[ci][1][id], pprev = p.dd[ci][2][id];
      double prev1 = p.d1[ci][1][id], pprev1 = p.d1[ci][2][id];
      double material = avg (mat, id);
      const double *om = p.omega, *ga = p.gamma;
      double omega, gamma;
      if (nmat == 2)
      {
        omega = (om[id + mo[0]] + om[id + mo[1]]) / 2.0;
        gamma = (ga[id + mo[0]] + ga[id + mo[1]]) / 2.0;
      }
      else
      {
        omega = (om[id + mo[0]] + om[id + mo[1]] + om[id + mo[2]] + om[id + mo[3]]) / 4.0;
        gamma = (ga[id + mo[0]] + ga[id + mo[1]] + ga[id + mo[2]] + ga[id + mo[3]]) / 4.0;
      }
      double sq = dt * omega;
      double A = 4 * mm * material + 2 * dt * mm * material * gamma + mm * (sq * sq);
      double b0 = (4 + 2 * dt * gamma) / A;
      double b1 = -8 / A;
      double b2 = (4 - 2 * dt * gamma) / A;
      double a1 = (2 * mm * (sq * sq) - 8 * mm * material) / A;
      double a2 = (4 * mm * material - 2 * dt * mm * material * gamma + mm * (sq * sq)) / A;
      p.d1[ci][0][id] = cur * b0 + prev * b1 + pprev * b2 - prev1 * a1 - pprev1 * a2;
    }
    double prev_eh = f1[id];
    double *const *src = META ? p.d1[ci] : p.dd[ci];
    double cur_db = src[0][id];
    double prev_db = src[1][id];
    double material1 = avg (mat, id);
    double modifier = material1 * mm;
    if (META)
      modifier = 1;
    const int q5 = pos[ax5], q4 = pos[ax4];
    double dd5 = t_dd5[q5];
    double ca2 = t_ca2[q5];
    double cb2 = (t_n4p[q4] / (modifier)) / dd5;
    double cc2 = (t_n4m[q4] / (modifier)) / dd5;
    f0[id] = prev_eh * ca2 + cur_db * cb2 - prev_db * cc2;
  }
}

// ------------------------------------------------- 3-D half-step by columns

// Incident value for the TF/SF slow path of plain_march_kernel (out of line:
// only the columns and planes on the faces take it).
__device__ __noinline__ double march_incident (const PlainHalf *p, int inc_len, int *err, int k, int x, int y, int z)
{
  return incident_value (p->g, p->inc, inc_len, err, k, x, y, z);
}

// E-from-D's two coefficients of a cell (out of line: the divisions are taken
// only where the material or a coefficient changes).
__device__ __noinline__ double2 march_coeffs (double plus, double minus, double modifier, double dd)
{
  const double p = (plus / modifier) / dd;
  return make_double2 (p, minus == plus ? p : (minus / modifier) / dd);
}

constexpr int kMarchBlock = 128;
constexpr int kMarchMax = 64;   // largest x chunk (per-plane TF/SF masks in shared memory)

// One half-step (all three components) of the FP64 plain form, 3-D: a thread
// owns one (y, z) column of a chunk of x planes and marches along x, the
// arithmetic of plain_component in its order.
//
// What bounds it: at one component per thread and cell (plain_fast_kernel)
// the half-step is bound by instructions, 410 per component and cell, most
// of them the four IEEE divisions of E-from-D, the index arithmetic and the
// reloads of the opposite family.  A column keeps all of that in registers:
//  * the y and z coefficients are constants of the thread, the x ones
//    uniform loads;
//  * E-from-D's coefficients are recomputed only when the averaged material
//    or an x coefficient changes from one plane to the next (two divisions,
//    four where sigma along the component's own axis differs from 0), so
//    uniform regions divide once per column;
//  * the x neighbours are the previous plane's values.
// Columns are numbered flat over y and z, so no lane idles on odd sizes; the
// next plane's material and coefficients are worked out after the stores,
// where few values are live (96 registers, 16 to 20 warps per SM).  What is left
// is memory latency (256^3: 11 to 13 of 16 warps wait for loads, 25 % issue
// active, 4.1 to 4.4 TB/s of DRAM; 512^3: 5.0 TB/s).
// 203 x 181 x 165, PML 12, TF/SF: 370 -> 210 us per half-step (a step 735 ->
// 429 us); a step at 80^3, PML 10: 82 -> 55 us.
// IS_H: the family, which orders the two differences of a curl.  LO: the lower
// cell of a difference (-1: E in E_CENTERED, H in H_CENTERED; 0 the other way
// round).  MK: material points a component averages (0: uniform 1, 1:
// per-component arrays of double material precision, 2 with LO = -1, 4 with
// LO = 0).
template <bool IS_H, int LO, bool PML, int MK>
__global__ void __launch_bounds__ (kMarchBlock, 5)
    plain_march_kernel (const __grid_constant__ PlainHalf p, const __grid_constant__ PlainTabs tb,
                        const __grid_constant__ IncidentJob inc, int inc_blocks, int col_blocks, int chunk, int inc_len,
                        int *err)
{
  if ((int) blockIdx.x < inc_blocks)
  {
    for (int i = blockIdx.x * kMarchBlock + threadIdx.x; i < inc.cells; i += inc_blocks * kMarchBlock)
    {
      if (p.is_h)
        inc.now[i] = inc.old[i] + (inc.other[i] - inc.other[i + 1]) * inc.modifier;
      else if (i == 0)
        inc.now[0] = *inc.src;
      else
        inc.now[i] = inc.old[i] + (inc.other[i - 1] - inc.other[i]) * inc.modifier;
    }
    return;
  }
  const GeomDev &g = p.g;
  const int b = (int) blockIdx.x - inc_blocks;
  const int wz = g.n[2] - 2, cols = (g.n[1] - 2) * wz;
  const int col = (b % col_blocks) * kMarchBlock + threadIdx.x;
  const int xa = 1 + (b / col_blocks) * chunk, xe = min (xa + chunk, g.n[0] - 1);

  // TF/SF terms (bit 4 ci + t) whose x range holds plane xa + i
  __shared__ unsigned s_terms[kMarchMax];
  if (p.use_tfsf)
  {
    for (int i = threadIdx.x; i < xe - xa; i += kMarchBlock)
    {
      unsigned m = 0;
      for (int ci = 0; ci < 3; ++ci)
        for (int t = 0; t < p.comp[ci].nterms; ++t)
          if (xa + i >= p.comp[ci].term[t].lo[0] && xa + i < p.comp[ci].term[t].hi[0])
            m |= 1u << (4 * ci + t);
      s_terms[i] = m;
    }
    __syncthreads ();
  }
  if (col >= cols)
    return;
  const int y = 1 + col / wz, z = 1 + col % wz;
  const int64_t sy = g.n[2], sx = (int64_t) g.n[1] * g.n[2];
  int64_t id = xa * sx + y * sy + z;
  unsigned terms = 0;   // terms whose y and z ranges hold the column
  if (p.use_tfsf)
    for (int ci = 0; ci < 3; ++ci)
      for (int t = 0; t < p.comp[ci].nterms; ++t)
      {
        const TermDev &tm = p.comp[ci].term[t];
        if (y >= tm.lo[1] && y < tm.hi[1] && z >= tm.lo[2] && z < tm.hi[2])
          terms |= 1u << (4 * ci + t);
      }

  const double dt = g.dt, dx = g.dx, mm = p.mat_modifier;
  // PML coefficients: component 0 has ca, cb along y, the denominator along
  // z, the numerators along x; 1 and 2 are its rotations
  // (the ones only march_coeffs takes are read there again)
  double ca0 = 1, cb0 = 0, e0 = 1, ca1 = 1, cb1 = 0, e2 = 1;
  if (PML)
  {
    ca0 = tb.t[0][0][y];
    cb0 = tb.t[0][1][y];
    e0 = tb.t[0][2][z];
    ca1 = tb.t[1][0][z];
    cb1 = tb.t[1][1][z];
    e2 = tb.t[2][2][y];
  }
  // what the current E-from-D coefficients (without PML: cb) were made from
  // (at first nothing: NaN differs from every material)
  const double none = __longlong_as_double (0x7ff8000000000000ll);
  double m_of[3] = {none, none, none}, np0 = 0, nm0 = 0, dd1 = 0;
  double cp[3] = {0, 0, 0}, cm[3] = {0, 0, 0};
  // x coefficients of the plane: component 2's ca, cb and component 1's ca2
  double cax = 1, cbx = 0, e1 = 1;
  auto coeffs = [&] (const double m[3], int x) __attribute__ ((always_inline)) {
    if (PML)
    {
      cax = tb.t[2][0][x];
      cbx = tb.t[2][1][x];
      e1 = tb.t[1][2][x];
      const double d = tb.t[1][3][x], a = tb.t[0][4][x], s = tb.t[0][5][x];
      if (m[0] != m_of[0] || a != np0 || s != nm0)
      {
        m_of[0] = m[0];
        np0 = a;
        nm0 = s;
        const double2 c = march_coeffs (a, s, m[0] * mm, tb.t[0][3][z]);
        cp[0] = c.x;
        cm[0] = c.y;
      }
      if (m[1] != m_of[1] || d != dd1)
      {
        m_of[1] = m[1];
        dd1 = d;
        const double2 c = march_coeffs (tb.t[1][4][y], tb.t[1][5][y], m[1] * mm, d);
        cp[1] = c.x;
        cm[1] = c.y;
      }
      if (m[2] != m_of[2])
      {
        m_of[2] = m[2];
        const double2 c = march_coeffs (tb.t[2][4][z], tb.t[2][5][z], m[2] * mm, tb.t[2][3][y]);
        cp[2] = c.x;
        cm[2] = c.y;
      }
    }
    else
    {
#pragma unroll
      for (int ci = 0; ci < 3; ++ci)
        if (m[ci] != m_of[ci])
        {
          m_of[ci] = m[ci];
          cp[ci] = dt / (m[ci] * mm * dx);
        }
    }
  };
  // material points of the plane at `id`, and those of the plane after it at
  // (0, 0), (y + 1), (z + 1) where the averages span x
  double mc = 1, my = 1, mz = 1, myz = 1, mx = 1, mxy = 1, mxz = 1;
  auto material = [&] (int64_t at) __attribute__ ((always_inline)) {
    if (MK == 1)
    {
      mc = p.matc[0][at];
      my = p.matc[1][at];
      mz = p.matc[2][at];
    }
    else if (MK == 2)
    {
      my = p.mat[at + sy];
      mz = p.mat[at + 1];
      mx = p.mat[at + sx];
    }
    else if (MK == 4)
    {
      myz = p.mat[at + sy + 1];
      mx = p.mat[at + sx];
      mxy = p.mat[at + sx + sy];
      mxz = p.mat[at + sx + 1];
    }
  };
  // their averages, then the plane's centre moves on
  auto averages = [&] (double m[3]) __attribute__ ((always_inline)) {
    m[0] = m[1] = m[2] = 1;
    if (MK == 1)
    {
      m[0] = mc;
      m[1] = my;
      m[2] = mz;
    }
    else if (MK == 2)
    {
      m[0] = (mc + mx) / 2.0;
      m[1] = (mc + my) / 2.0;
      m[2] = (mc + mz) / 2.0;
      mc = mx;
    }
    else if (MK == 4)
    {
      m[0] = ((mc + mz) / 2.0 + (my + myz) / 2.0) / 2.0;
      m[1] = ((mc + mz) / 2.0 + (mx + mxz) / 2.0) / 2.0;
      m[2] = ((mc + my) / 2.0 + (mx + mxy) / 2.0) / 2.0;
      mc = mx;
      my = mxy;
      mz = mxz;
    }
  };

  const double *O0 = p.opp[0], *O1 = p.opp[1], *O2 = p.opp[2];
  // carried along x: LO = -1 the previous plane's values (the x neighbours),
  // LO = 0 the centre's (read a plane ahead as its x neighbours)
  double c1 = O1[LO ? id - sx : id], c2 = O2[LO ? id - sx : id];
  if (MK == 2 || MK == 4)
    mc = p.mat[id];
  if (MK == 4)
  {
    my = p.mat[id + sy];
    mz = p.mat[id + 1];
  }
  {
    double m[3];
    material (id);
    averages (m);
    coeffs (m, xa);
  }
  for (int x = xa; x < xe; ++x, id += sx)
  {
    const int64_t oy = LO ? id - sy : id + sy, oz = LO ? id - 1 : id + 1;
    const double o0 = O0[id];
    const double n1 = O1[LO ? id : id + sx], n2 = O2[LO ? id : id + sx];
    const double o2y = O2[oy], o1z = O1[oz], o0z = O0[oz], o0y = O0[oy];
    double old[3], fld[3] = {0, 0, 0};
#pragma unroll
    for (int ci = 0; ci < 3; ++ci)
    {
      old[ci] = PML ? p.dd[ci][1][id] : p.f[ci][1][id];
      if (PML)
        fld[ci] = p.f[ci][1][id];
    }
    // (the next plane's material and coefficients follow the stores, where
    // no field value is live; its loads are in flight with the fields')
    if (x + 1 < xe)
      material (id + sx);
    // neighbours of the curls, v[ci] = {11, 12, 21, 22}: the difference of the
    // family's component ci + 2 along ci + 1 and of ci + 1 along ci + 2, in
    // this order for E, in the other for H
    double v[3][4];
    auto pair = [&] (int ci, int q, double near, double far) {
      const int at = (q == 0) != IS_H ? 0 : 2;
      v[ci][at] = LO ? far : near;
      v[ci][at + 1] = LO ? near : far;
    };
    const double x1 = LO ? c1 : n1, x2 = LO ? c2 : n2, o1 = LO ? n1 : c1, o2 = LO ? n2 : c2;
    pair (0, 0, o2, o2y);
    pair (0, 1, o1, o1z);
    pair (1, 0, o0, o0z);
    pair (1, 1, o2, x2);
    pair (2, 0, o1, x1);
    pair (2, 1, o0, o0y);
    c1 = n1;
    c2 = n2;
    if (p.use_tfsf)
    {
      const unsigned on = terms & s_terms[x - xa];
      for (unsigned left = on; left; left &= left - 1)
      {
        const int bit = __ffs ((int) left) - 1, ci = bit >> 2;
        const TermDev &tm = p.comp[ci].term[bit & 3];
        double diff = march_incident (&p, inc_len, err, tm.inc_comp, x + tm.aux[0], y + tm.aux[1], z + tm.aux[2]);
        if (tm.negate < 0)
          diff *= -1.0;
        const int at = 4 * ci + tm.slot;
#pragma unroll
        for (int q = 0; q < 12; ++q)
          if (at == q)
            v[q / 4][q % 4] -= diff;
      }
    }
    const double ca[3] = {ca0, ca1, cax}, cb[3] = {PML ? cb0 : cp[0], PML ? cb1 : cp[1], PML ? cbx : cp[2]};
    const double e[3] = {e0, e1, e2};
#pragma unroll
    for (int ci = 0; ci < 3; ++ci)
    {
      const double tmp = v[ci][1] - v[ci][0] - v[ci][3] + v[ci][2];
      const double nv = old[ci] * ca[ci] + tmp * cb[ci];
      if (PML)
      {
        p.dd[ci][0][id] = nv;
        p.f[ci][0][id] = fld[ci] * e[ci] + nv * cp[ci] - old[ci] * cm[ci];
      }
      else
        p.f[ci][0][id] = nv;
    }
    if (x + 1 < xe)
    {
      double m[3];
      averages (m);
      coeffs (m, x + 1);
    }
  }
}

int launch_plain_tables (const PlainHalf &p, double *const out[3][6], cudaStream_t s)
{
  PlainTabOut o;
  for (int ci = 0; ci < 3; ++ci)
    for (int j = 0; j < 6; ++j)
      o.t[ci][j] = out[ci][j];
  plain_tables_kernel<<<dim3 (4, 3, 3), 256, 0, s>>> (p, o);
  return 1;
}

int launch_plain_fast (const PlainHalf &p, const PlainTabs &t, int inc_len, int *err, int sm_count,
                       cudaStream_t s)
{
  const int ix = (p.g.drop & 1) ? 1 : p.g.n[0] - 2;
  const int iy = (p.g.drop & 2) ? 1 : p.g.n[1] - 2;
  const int iz = (p.g.drop & 4) ? 1 : p.g.n[2] - 2;
  int64_t total = (int64_t) ix * iy * iz;
  int64_t blocks = (total + 255) / 256;
  int64_t cap = (int64_t) sm_count * 8 * 16;
  if (blocks > cap)
    blocks = cap;
  if (blocks < 1)
    blocks = 1;
  int ncomp = 0;
  for (int ci = 0; ci < 3; ++ci)
    ncomp += p.comp[ci].exists ? 1 : 0;
  if (ncomp == 0)
    return 0;
  auto kern = p.use_pml ? (p.use_meta ? (p.use_tfsf ? plain_fast_kernel<true, true, true>
                                                    : plain_fast_kernel<true, true, false>)
                                      : (p.use_tfsf ? plain_fast_kernel<true, false, true>
                                                    : plain_fast_kernel<true, false, false>))
                        : (p.use_tfsf ? plain_fast_kernel<false, false, true> : plain_fast_kernel<false, false, false>);
  kern<<<(unsigned) (blocks * ncomp), 256, 0, s>>> (p, t, ncomp, inc_len, err);
  return 1;
}

int launch_plain_march (const PlainHalf &p, const PlainTabs &t, const IncidentJob &inc, bool mat_uniform, int inc_len,
                        int *err, int sm_count, cudaStream_t s)
{
  const int cols = (p.g.n[1] - 2) * (p.g.n[2] - 2), planes = p.g.n[0] - 2;
  const int col_blocks = (cols + kMarchBlock - 1) / kMarchBlock;
  const int inc_blocks = inc.cells > 0 ? std::min (64, (inc.cells + kMarchBlock - 1) / kMarchBlock) : 0;
  const int mk = mat_uniform ? 0 : (p.dmp ? 1 : p.comp[0].nmat);
  using Kernel = void (*) (const PlainHalf, const PlainTabs, const IncidentJob, int, int, int, int, int *);
#define FDTDB_MARCH(H, LO, PML)                                                                                        \
  (mk == 0 ? plain_march_kernel<H, LO, PML, 0> : mk == 1 ? plain_march_kernel<H, LO, PML, 1>                           \
                                                         : plain_march_kernel<H, LO, PML, (LO ? 2 : 4)>)
  const bool low = p.comp[0].d11[1] < 0 || p.comp[0].d11[2] < 0;   // (E differs along y first, H along z)
  Kernel kern = nullptr;
  if (p.is_h)
    kern = low ? (p.use_pml ? FDTDB_MARCH (true, -1, true) : FDTDB_MARCH (true, -1, false))
               : (p.use_pml ? FDTDB_MARCH (true, 0, true) : FDTDB_MARCH (true, 0, false));
  else
    kern = low ? (p.use_pml ? FDTDB_MARCH (false, -1, true) : FDTDB_MARCH (false, -1, false))
               : (p.use_pml ? FDTDB_MARCH (false, 0, true) : FDTDB_MARCH (false, 0, false));
#undef FDTDB_MARCH
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor (&per_sm, kern, kMarchBlock, 0) != cudaSuccess || per_sm < 1)
    per_sm = 4;
  // x chunk: the blocks run in waves of sm_count * per_sm, each as long as
  // its planes and the start of a column (about three planes' time)
  int chunk = 4;
  double best = 1e300;
  for (int c : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64})
  {
    const int m = (planes + c - 1) / c, even = (planes + m - 1) / m;
    const double waves = std::max (1.0, (double) col_blocks * m / ((double) sm_count * per_sm));
    const double cost = (waves < 8 ? std::ceil (waves) : waves + 0.5) * (even + 3);
    if (cost < best * 0.999)
    {
      best = cost;
      chunk = even;
    }
  }
  const int chunks = (planes + chunk - 1) / chunk;
  kern<<<(unsigned) (inc_blocks + col_blocks * chunks), kMarchBlock, 0, s>>> (p, t, inc, inc_blocks, col_blocks, chunk,
                                                                              inc_len, err);
  return 1;
}

int launch_plain_half (const PlainHalf &p, int inc_len, int *err, int sm_count, cudaStream_t s)
{
  const int ix = (p.g.drop & 1) ? 1 : p.g.n[0] - 2;
  const int iy = (p.g.drop & 2) ? 1 : p.g.n[1] - 2;
  const int iz = (p.g.drop & 4) ? 1 : p.g.n[2] - 2;
  int64_t total = (int64_t) ix * iy * iz;
  int64_t blocks = (total + 255) / 256;
  int64_t cap = (int64_t) sm_count * 8 * 16;
  if (blocks > cap)
    blocks = cap;
  if (blocks < 1)
    blocks = 1;
  if (p.dmp)
  {
    if (p.cs_mask)
      plain_half_kernel<true, true><<<(unsigned) blocks, 256, 0, s>>> (p, inc_len, err);
    else
      plain_half_kernel<true, false><<<(unsigned) blocks, 256, 0, s>>> (p, inc_len, err);
  }
  else if (p.cs_mask)
    plain_half_kernel<false, true><<<(unsigned) blocks, 256, 0, s>>> (p, inc_len, err);
  else
    plain_half_kernel<false, false><<<(unsigned) blocks, 256, 0, s>>> (p, inc_len, err);
  return 1;
}

int launch_incident_e (const IncidentJob &j, cudaStream_t s)
{
  incident_e_kernel<<<(j.cells + 255) / 256, 256, 0, s>>> (j);
  return 1;
}

int launch_incident_h (const IncidentJob &j, cudaStream_t s)
{
  incident_h_kernel<<<(j.cells + 255) / 256, 256, 0, s>>> (j);
  return 1;
}

int launch_incident (const IncidentPair &j, cudaStream_t s)
{
  incident_kernel<<<(std::max (j.e.cells, j.h.cells) + 255) / 256, 256, 0, s>>> (j);
  return 1;
}

int launch_point_source (double *f, size_t index, const double *src, int src_index, cudaStream_t s)
{
  point_source_kernel<<<1, 32, 0, s>>> (f, index, src, src_index);
  return 1;
}

__global__ void fine_average_kernel (const double *fine, double *out64, float *out32, FineAvg a)
{
  const int64_t total = (int64_t) a.n[0] * a.n[1] * a.n[2];
  for (int64_t id = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; id < total;
       id += (int64_t) gridDim.x * blockDim.x)
  {
    const int z = (int) (id % a.n[2]);
    const int64_t r = id / a.n[2];
    const int y = (int) (r % a.n[1]);
    const int x = (int) (r / a.n[1]);
    const int p[3] = {x, y, z};
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
    {
      // the outer shell's last cell would reach one fine cell past the grid;
      // its material is never used, so clamp
      int q[3];
#pragma unroll
      for (int b = 0; b < 3; ++b)
        q[b] = min (a.mul[b] * p[b] + a.off[j][b], a.nf[b] - 1);
      v[j] = fine[((int64_t) q[0] * a.nf[1] + q[1]) * a.nf[2] + q[2]];
    }
    // ((v1 + v2) / 2 + (v3 + v4) / 2) / 2, twice, then / 2
    const double lo = ((v[0] + v[1]) / 2.0 + (v[2] + v[3]) / 2.0) / 2.0;
    const double hi = ((v[4] + v[5]) / 2.0 + (v[6] + v[7]) / 2.0) / 2.0;
    const double m = (lo + hi) / 2.0;
    if (out64)
      out64[id] = m;
    if (out32)
      out32[id] = (float) m;
  }
}

// Scattered field for a dump (Scheme::makeGridScattered, Source/Scheme/
// Scheme.inc.h:4113-4226): inside the TF/SF box (real coordinates within
// [left, right] on every kept axis) the component minus its incident value.
__global__ void scattered_kernel (double *f, GeomDev g, int k, const double *inc, int inc_len, double3 left,
                                  double3 right, int *err)
{
  const int64_t total = (int64_t) g.n[0] * g.n[1] * g.n[2];
  const double lo[3] = {left.x, left.y, left.z}, hi[3] = {right.x, right.y, right.z};
  for (int64_t id = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; id < total;
       id += (int64_t) gridDim.x * blockDim.x)
  {
    const int z = (int) (id % g.n[2]);
    const int64_t r = id / g.n[2];
    const int y = (int) (r % g.n[1]);
    const int x = (int) (r / g.n[1]);
    const int p[3] = {x, y, z};
    bool inside = true;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      const double c = (double) p[a] + g.min_fp[k][a];
      if (!((g.drop >> a) & 1) && (c < lo[a] || c > hi[a]))
        inside = false;
    }
    if (inside)
      f[id] = f[id] - incident_value (g, inc, inc_len, err, k, x, y, z);
  }
}

int launch_scattered (double *f, const GeomDev &g, int k, const double *inc, int inc_len, const double left[3],
                      const double right[3], int *err, int sm_count, cudaStream_t s)
{
  scattered_kernel<<<sm_count * 4, 256, 0, s>>> (f, g, k, inc, inc_len, make_double3 (left[0], left[1], left[2]),
                                                 make_double3 (right[0], right[1], right[2]), err);
  return 1;
}

int launch_fine_average (const double *fine, double *out64, float *out32, const FineAvg &a, int sm_count,
                         cudaStream_t s)
{
  fine_average_kernel<<<sm_count * 4, 256, 0, s>>> (fine, out64, out32, a);
  return 1;
}

}  // namespace fdtdb
