// tmz_batch.cu - many 2-D TMz simulations of uneven sizes in one persistent
// kernel launch (captured in a CUDA graph), FP32; calls of a few steps in a
// launch per step.
//
// Every instance is an fdtd3d Dim2_TMz E_CENTERED run (Ez, Hx, Hy) with PML,
// its own eps map and a point source at its centre; they share dx, Courant
// factor, PML width and source.  The formulation per instance is the FP32
// form of fast_kernels.cu (H stored as eta0*H, PML auxiliaries only in PML
// cells); the step semantics are the reference's (no field update at t = 0,
// Source/Scheme/Scheme.inc.h:1032; hard point source after the E update).
//
// Work decomposition: a work list of tiles, largest instance first, taken by
// persistent CTAs from an atomic counter.  A round advances every tile up to
// kTileSteps steps (tile2d.cuh: own cells and halo in registers and shared
// memory, the halo recomputed), fields double buffered; a grid-wide barrier
// separates rounds.  One step per round (a warp per 30-cell strip, fields
// streamed from L2 / HBM) was bound by bytes in flight and the barrier: 20
// instances, 6.08 M cells: 82 us per step, 49 us now.  Calls of up to three
// steps go by cells instead, a launch per step (tmz_cells_kernel).
// The barrier is a bounded spin on a global generation counter (globaltimer
// timeout -> error flag, every CTA leaves); the kernel is launched
// cooperatively so all CTAs are co-resident.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/fdtd_b200.h"
#include "kernels.h"
#include "setup.h"
#include "tile2d.cuh"

namespace fdtdb {

namespace {

constexpr double kEta0B = 376.730313461770655;

struct InstDev
{
  long long off;                      // first cell of the instance in every arena
  int nx, ny;
  int tab;                            // first entry of the instance's 1-D tables
  int ilo[3][2], ihi[3][2];           // per component (Ez, Hx, Hy): sigma == 0 range in x, y
  int ps;                             // 1: point source at the centre
};

// per instance, 12 tables laid out back to back:
//   Ez: ca1(x) sq1(x) p5(y) q5(y)    Hx: g4p(x) g4m(x) ca1(y) sq1(y)    Hy: p5(x) q5(x) g4p(y) g4m(y)
// each of length nx or ny, in that order; the pairs along the dropped axis
// are the six identity values at the head of the array

struct TileDev
{
  int inst, u0, v0;                   // corner of the tile, halo included
};

// A CTA's part of a step by cells: kCellRows rows from u0, kCellCols columns
// from v0.
struct PatchDev
{
  int inst, u0, v0;
};
constexpr int kCellWarps = 8, kCellRun = 4, kCellRows = kCellWarps * kCellRun, kCellCols = 31;

struct BatchParams
{
  const Tile2D *inst[2];              // per instance, buffer set 0 / 1 as the current one
  const TileDev *tiles;
  int ntiles, ninst;
  const double *src;                  // E source value per step of this launch, from [1]
  unsigned *counters;                 // [0], [1]: tile counters by round parity; [2]: barrier arrivals
  unsigned *generation;
  int *err;
  long long timeout_ns;
  // per launch
  unsigned t_start;
  unsigned nsteps;
  int cur;                            // buffer set holding the current time level
};

__device__ __forceinline__ long long globaltimer ()
{
  long long t;
  asm volatile ("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier with a time limit.  Returns false if any CTA gave up.
__device__ bool grid_barrier (const BatchParams &p)
{
  __shared__ int ok;
  __syncthreads ();
  if (threadIdx.x == 0 && threadIdx.y == 0)
  {
    volatile unsigned *gen = p.generation;
    unsigned g = *gen;
    __threadfence ();
    unsigned arrived = atomicAdd (&p.counters[2], 1u);
    if (arrived == gridDim.x - 1)
    {
      atomicExch (&p.counters[2], 0u);
      __threadfence ();
      atomicAdd ((unsigned *) p.generation, 1u);
    }
    else
    {
      long long t0 = globaltimer ();
      while (*gen == g)
      {
        if (*((volatile int *) p.err) != 0 || globaltimer () - t0 > p.timeout_ns)
        {
          atomicExch (p.err, 2);
          break;
        }
        __nanosleep (64);
      }
    }
    __threadfence ();
    ok = *((volatile int *) p.err) == 0;
  }
  __syncthreads ();
  return ok != 0;
}

template <int CU, int CV>
__global__ void __launch_bounds__ (kTileThreads, 1) tmz_batch_kernel (BatchParams p)
{
  extern __shared__ __align__ (16) unsigned char tile_smem[];
  __shared__ double s_inc[2][kTileThreads];
  __shared__ Tile2D s_p;
  __shared__ int s_tile;
  const int tid = threadIdx.x + 32 * threadIdx.y;
  int cur = p.cur;
  unsigned s = 0;
  if (p.t_start == 0)
  {
    // no field update at t = 0; the hard source still sets Ez
    if (blockIdx.x == 0)
      for (int i = tid; i < p.ninst; i += kTileThreads)
      {
        const Tile2D &q = p.inst[cur][i];
        if (q.comp[0].source)
          ((float *) q.comp[0].in)[(long long) q.pu * q.nv + q.pv] = (float) p.src[1];
      }
    if (!grid_barrier (p))
      return;
    s = 1;
  }
  for (unsigned round = 0; s < p.nsteps; ++round)
  {
    const int steps = (int) min ((unsigned) kTileSteps, p.nsteps - s);
    for (;;)
    {
      __syncthreads ();   // (the previous tile's shared values have been used)
      if (tid == 0)
        s_tile = (int) atomicAdd (&p.counters[round & 1], 1u);
      __syncthreads ();
      if (s_tile >= p.ntiles)
        break;
      const TileDev t = p.tiles[s_tile];
      const unsigned *from = reinterpret_cast<const unsigned *> (p.inst[cur] + t.inst);
      for (int q = tid; q < (int) (sizeof (Tile2D) / 4); q += kTileThreads)
        reinterpret_cast<unsigned *> (&s_p)[q] = from[q];
      __syncthreads ();
      if (tid == 0)
      {
        s_p.steps = steps;
        s_p.src = p.src + s;
      }
      __syncthreads ();
      tile2d_steps<float, float, CU, CV, 0, false> (s_p, t.u0, t.v0, tile_smem, s_inc);
    }
    // the counter of the next round (same parity as the previous one) is idle now
    if (blockIdx.x == 0 && tid == 0)
      atomicExch (&p.counters[(round + 1) & 1], 0u);
    if (!grid_barrier (p))
      return;
    cur ^= 1;
    s += steps;
  }
}

// The arenas of a step by cells: Ez, Hx, Hy and their auxiliaries, from one set
// into the other.
struct CellArrays
{
  const float *in[3], *xin[3];
  float *out[3], *xout[3];
  const float *eps, *tab;
  float courant;
  int use_pml;
};

// F after a curl of `cu` (m: 1 / eps or 1), and X where the cell has PML.
__device__ __forceinline__ float cell_update (bool pml, float f, float cu, float m, float S, float ca1, float sq1,
                                              float p5, float q5, float g4p, float g4m, const float *xo, float *xn,
                                              int64_t id, bool store)
{
  if (!pml)
    return f + S * m * cu;
  const float o = xo[id], n = ca1 * o + sq1 * cu;
  if (store)
    xn[id] = n;
  return p5 * f + (g4p * n - g4m * o) * q5 * m;
}

// One time step of every instance (update = 0: only the sources): a thread Ez of
// four cells of a column and, again, of the one after them, then H of the four;
// Ez of the next column by a shuffle (lane 31 has no cell of its own).  No
// thread waits for another, and every value is read and written once.  The form
// of calls of a few steps, whose tiles would be set up, read and written for
// little.
__global__ void __launch_bounds__ (32 * kCellWarps)
    tmz_cells_kernel (const __grid_constant__ CellArrays p, const InstDev *inst, const PatchDev *patches,
                      const double *src, int update)
{
  const PatchDev td = patches[blockIdx.x];
  const InstDev &in = inst[td.inst];
  const int nx = in.nx, ny = in.ny, v = td.v0 + threadIdx.x, u0 = td.u0 + kCellRun * threadIdx.y;
  const int64_t base = in.off + (int64_t) u0 * ny + v;
  const int su = in.ps && v == ny / 2 ? nx / 2 : -1;
  if (!update)
  {
    if (threadIdx.x < kCellCols && su >= u0 && su < u0 + kCellRun)
      const_cast<float *> (p.in[0])[base + (int64_t) (su - u0) * ny] = (float) *src;
    return;
  }
  if (u0 > nx - 2)
    return;   // (the whole warp)
  const float S = p.courant;
  const bool pml = p.use_pml, column = v <= ny - 2, own = column && threadIdx.x < kCellCols;
  // tables of the instance: Ez ca1, sq1 (x), p5, q5 (y); Hx g4p, g4m (x), ca1,
  // sq1 (y); Hy p5, q5 (x), g4p, g4m (y)
  const float *const T = p.tab + in.tab;
  const int t1 = 2 * (nx + ny), t2 = 2 * t1;
  float e[kCellRun + 1], hx[kCellRun + 1], hy[kCellRun + 2], left[kCellRun + 1], m[kCellRun + 1];
  hy[0] = column ? p.in[2][base - ny] : 0.f;
#pragma unroll
  for (int r = 0; r <= kCellRun; ++r)
  {
    const int64_t id = base + (int64_t) r * ny;
    const bool there = v <= ny - 1 && u0 + r <= nx - 1, on = column && u0 + r <= nx - 2;
    e[r] = there ? p.in[0][id] : 0.f;
    hx[r] = on ? p.in[1][id] : 0.f;
    left[r] = on ? p.in[1][id - 1] : 0.f;
    hy[r + 1] = on ? p.in[2][id] : 0.f;
    m[r] = on ? p.eps[id] : 1.f;
  }
  {
    const bool yin = v >= in.ilo[0][1] && v < in.ihi[0][1];
    const int lo = in.ilo[0][0], hi = in.ihi[0][0];
#pragma unroll
    for (int r = 0; r <= kCellRun; ++r)
    {
      const int u = u0 + r;
      if (!column || u > nx - 2)
        continue;
      const int64_t id = base + (int64_t) r * ny;
      const bool pm = pml && !(yin && u >= lo && u < hi), store = own && r < kCellRun;
      e[r] = cell_update (pm, e[r], (hy[r + 1] - hy[r]) - (hx[r] - left[r]), 1.f / m[r], S, pm ? T[u] : 1.f,
                          pm ? T[nx + u] : S, pm ? T[2 * nx + v] : 1.f, pm ? T[2 * nx + ny + v] : 1.f, 1.f, 1.f,
                          p.xin[0], p.xout[0], id, store);
      if (u == su)
        e[r] = (float) *src;
      if (store)
        p.out[0][id] = e[r];
    }
  }
  const bool yx = v >= in.ilo[1][1] && v < in.ihi[1][1], yy = v >= in.ilo[2][1] && v < in.ihi[2][1];
  const int xlo = in.ilo[1][0], xhi = in.ihi[1][0], ylo = in.ilo[2][0], yhi = in.ihi[2][0];
#pragma unroll
  for (int r = 0; r < kCellRun; ++r)
  {
    const int u = u0 + r;
    const float up = __shfl_down_sync (0xffffffffu, e[r], 1);
    if (!own || u > nx - 2)
      continue;
    const int64_t id = base + (int64_t) r * ny;
    const bool px = pml && !(yx && u >= xlo && u < xhi), py = pml && !(yy && u >= ylo && u < yhi);
    p.out[1][id] = cell_update (px, hx[r], e[r] - up, 1.f, S, px ? T[t1 + 2 * nx + v] : 1.f,
                                px ? T[t1 + 2 * nx + ny + v] : S, 1.f, 1.f, px ? T[t1 + u] : 1.f,
                                px ? T[t1 + nx + u] : 1.f, p.xin[1], p.xout[1], id, true);
    p.out[2][id] = cell_update (py, hy[r + 1], e[r + 1] - e[r], 1.f, S, 1.f, S, py ? T[t2 + u] : 1.f,
                                py ? T[t2 + nx + u] : 1.f, py ? T[t2 + 2 * nx + v] : 1.f,
                                py ? T[t2 + 2 * nx + ny + v] : 1.f, p.xin[2], p.xout[2], id, true);
  }
}

}  // namespace

}  // namespace fdtdb

// --------------------------------------------------------------------------
// host side

struct fdtd_batch
{
  int device = 0;
  int sm_count = 148;
  cudaStream_t stream = nullptr;
  fdtd_config base;
  std::vector<fdtdb::Geometry> geo;
  std::vector<fdtdb::InstDev> inst;
  long long cells = 0;
  int ntab = 0;
  std::vector<float> tab_host;
  fdtdb::Tile2D *d_inst[2] = {};
  double *stage = nullptr;            // FP64 copy of one component on its way to the host
  size_t stage_cells = 0;
  fdtdb::TileDev *d_tiles = nullptr;
  int ntiles = 0;
  fdtdb::PatchDev *d_patches = nullptr;
  fdtdb::InstDev *d_geo = nullptr;
  int npatches = 0;
  float *d_tab = nullptr;
  float *ez[2] = {}, *hx[2] = {}, *hy[2] = {}, *aez[2] = {}, *ahx[2] = {}, *ahy[2] = {};
  float *eps = nullptr;
  double *d_src = nullptr, *h_src = nullptr;
  size_t src_cap = 0;
  unsigned *d_counters = nullptr;
  unsigned *d_generation = nullptr;
  int *d_err = nullptr;
  int cur = 0;
  // launch shape of the tiles (autotuned): tile height in x (64: 64 x 64 cells, 32: 32 x
  // 32, halo included), CTAs per SM
  bool tuning = false;                // every call in tiles
  int x_chunk = 64;
  int ctas_per_sm = 1;
  // graph of (source upload, counter reset, persistent kernel)
  cudaGraphExec_t graph = nullptr;
  unsigned graph_steps = 0;
  unsigned graph_t = 0;
  int graph_cur = -1;
  bool use_graph = true;
  bool graph_ok = false;
  double last_ms = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  long long wait_limit_ns = 0;        // grid-barrier wait limit (<= 0: 5 s)
  std::string err;
  std::vector<void *> allocs;
};

namespace {

using fdtdb::BatchParams;

int bfail (fdtd_batch *b, int code, const std::string &m)
{
  if (b)
    b->err = m;
  return code;
}

#define BCK(call)                                                                                  \
  do                                                                                               \
  {                                                                                                \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess)                                                                         \
      return bfail (b, e_ == cudaErrorMemoryAllocation ? FDTD_ERR_NOMEM : FDTD_ERR_CUDA,           \
                    std::string (#call) + ": " + cudaGetErrorString (e_));                          \
  } while (0)

int balloc (fdtd_batch *b, void **p, size_t bytes)
{
  cudaError_t e = fdtdb::device_malloc (p, bytes ? bytes : 16);
  if (e != cudaSuccess)
    return bfail (b, FDTD_ERR_NOMEM, std::string ("cudaMalloc: ") + cudaGetErrorString (e));
  b->allocs.push_back (*p);
  e = cudaMemsetAsync (*p, 0, bytes ? bytes : 16, b->stream);
  return e == cudaSuccess ? FDTD_OK : bfail (b, FDTD_ERR_CUDA, cudaGetErrorString (e));
}

#define BALLOC(ptr, bytes)                                                                         \
  do                                                                                               \
  {                                                                                                \
    int r_ = balloc (b, (void **) &(ptr), (bytes));                                                \
    if (r_ != FDTD_OK)                                                                             \
      return r_;                                                                                   \
  } while (0)

int build_tiles (fdtd_batch *b, int x_chunk)
{
  std::vector<fdtdb::TileDev> tiles;
  // large instances first so the atomic work queue ends on small tiles
  std::vector<int> order (b->inst.size ());
  for (size_t i = 0; i < order.size (); ++i)
    order[i] = (int) i;
  std::sort (order.begin (), order.end (), [&] (int a, int c) {
    return (long long) b->inst[a].nx * b->inst[a].ny > (long long) b->inst[c].nx * b->inst[c].ny;
  });
  for (int i : order)
  {
    const fdtdb::InstDev &in = b->inst[i];
    const int own = x_chunk - 2 * fdtdb::kTileSteps;
    for (int u = 0; u < in.nx; u += own)
      for (int v = 0; v < in.ny; v += own)
        tiles.push_back ({i, u - fdtdb::kTileSteps, v - fdtdb::kTileSteps});
  }
  if (b->d_tiles)
  {
    auto it = std::find (b->allocs.begin (), b->allocs.end (), (void *) b->d_tiles);
    if (it != b->allocs.end ())
      b->allocs.erase (it);
    BCK (cudaStreamSynchronize (b->stream));
    cudaFree (b->d_tiles);
    b->d_tiles = nullptr;
  }
  BALLOC (b->d_tiles, tiles.size () * sizeof (fdtdb::TileDev));
  BCK (cudaMemcpyAsync (b->d_tiles, tiles.data (), tiles.size () * sizeof (fdtdb::TileDev), cudaMemcpyHostToDevice,
                        b->stream));
  BCK (cudaStreamSynchronize (b->stream));
  b->ntiles = (int) tiles.size ();
  b->x_chunk = x_chunk;
  return FDTD_OK;
}

void drop_graph (fdtd_batch *b)
{
  if (b->graph)
    cudaGraphExecDestroy (b->graph);
  b->graph = nullptr;
  b->graph_steps = 0;
  b->graph_cur = -1;
}

BatchParams params (fdtd_batch *b, uint32_t t_start, uint32_t n)
{
  BatchParams p;
  std::memset (&p, 0, sizeof (p));
  p.inst[0] = b->d_inst[0];
  p.inst[1] = b->d_inst[1];
  p.ninst = (int) b->inst.size ();
  p.tiles = b->d_tiles;
  p.ntiles = b->ntiles;
  p.src = b->d_src;
  p.counters = b->d_counters;
  p.generation = b->d_generation;
  p.err = b->d_err;
  p.timeout_ns = b->wait_limit_ns > 0 ? b->wait_limit_ns : 5000000000LL;
  p.t_start = t_start;
  p.nsteps = n;
  p.cur = b->cur;
  return p;
}

// The kernel of a tile height and its shared memory.
const void *batch_kernel (int tile, int &smem)
{
  using fdtdb::TileMem;
  if (tile == 32)
  {
    smem = TileMem<float, 2, 1>::BYTES;
    return (const void *) fdtdb::tmz_batch_kernel<2, 1>;
  }
  smem = TileMem<float, 4, 2>::BYTES;
  return (const void *) fdtdb::tmz_batch_kernel<4, 2>;
}

// co-resident CTAs per SM (0: the kernel does not fit)
int max_ctas (int tile)
{
  int per_sm = 0, smem = 0;
  const void *k = batch_kernel (tile, smem);
  if (cudaFuncSetAttribute (k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor (&per_sm, k, fdtdb::kTileThreads, smem) != cudaSuccess)
  {
    cudaGetLastError ();
    return 0;
  }
  return per_sm;
}

// Whether a call of n steps takes them by cells (tmz_cells_kernel).  us per
// call of 1, 2, 3, 4, 5 steps, PML, cells / tiles: one instance of 512^2 25 / 38,
// 34 / 40, 44 / 42, 52 / 45, 64 / 48; 20 of 100 .. 1000 a side (4.5 M cells) 69 /
// 206, 120 / 220, 173 / 235, 223 / 251, 277 / 265; two of 2048^2 87 / 312, 157 /
// 332, 230 / 351, 299 / 372, 373 / 392.
bool by_cells (const fdtd_batch *b, uint32_t n)
{
  return n <= 3 && !b->tuning;
}

// Enqueues one call (source upload, then counter reset and cooperative kernel,
// or the steps by cells).
int enqueue (fdtd_batch *b, uint32_t t_start, uint32_t n)
{
  BCK (cudaMemcpyAsync (b->d_src + 1, b->h_src, (size_t) n * sizeof (double), cudaMemcpyHostToDevice, b->stream));
  if (by_cells (b, n))
  {
    int cur = b->cur;
    for (uint32_t s = 0; s < n; ++s)
    {
      const int o = cur, w = 1 - cur, update = t_start + s > 0;
      const fdtdb::CellArrays p = {{b->ez[o], b->hx[o], b->hy[o]},
                                   {b->aez[o], b->ahx[o], b->ahy[o]},
                                   {b->ez[w], b->hx[w], b->hy[w]},
                                   {b->aez[w], b->ahx[w], b->ahy[w]},
                                   b->eps,
                                   b->d_tab,
                                   b->tab_host[1],
                                   b->base.use_pml};
      fdtdb::tmz_cells_kernel<<<b->npatches, dim3 (32, fdtdb::kCellWarps), 0, b->stream>>> (
          p, b->d_geo, b->d_patches, b->d_src + 1 + s, update);
      cur ^= update;
    }
    BCK (cudaGetLastError ());
    return FDTD_OK;
  }
  BCK (cudaMemsetAsync (b->d_counters, 0, 3 * sizeof (unsigned), b->stream));
  BatchParams p = params (b, t_start, n);
  void *args[] = {&p};
  int ctas = std::min (b->ctas_per_sm, max_ctas (b->x_chunk)) * b->sm_count;
  if (ctas <= 0)
    return bfail (b, FDTD_ERR_CUDA, "batch kernel does not fit on the device");
  int smem = 0;
  const void *kern = batch_kernel (b->x_chunk, smem);
  cudaLaunchConfig_t lc;
  std::memset (&lc, 0, sizeof (lc));
  lc.gridDim = dim3 (ctas);
  lc.blockDim = dim3 (32, fdtdb::kTileWarps);
  lc.dynamicSmemBytes = smem;
  lc.stream = b->stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  lc.attrs = &attr;
  lc.numAttrs = 1;
  BCK (cudaLaunchKernelExC (&lc, kern, args));
  return FDTD_OK;
}

// Cells of the read-out's staging buffer at most (64 MB; no row is longer).
constexpr size_t kStageCells = (size_t) 1 << 23;

// Rounds of a call (by cells: its steps): the buffer set changes with each.
uint32_t batch_rounds (const fdtd_batch *b, uint32_t t_start, uint32_t n)
{
  const uint32_t steps = n - (t_start == 0 ? 1 : 0);
  return by_cells (b, n) ? steps : (steps + fdtdb::kTileSteps - 1) / fdtdb::kTileSteps;
}

}  // namespace

namespace fdtdb {
namespace {

__global__ void fill_float_kernel (float *p, size_t n, float v)
{
  for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t) gridDim.x * blockDim.x)
    p[i] = v;
}

}  // namespace
}  // namespace fdtdb

namespace {

int create_batch (fdtd_batch *b, const fdtd_config *base, int count, const int *sizes, int device)
{
  using namespace fdtdb;
  if (base->mode != FDTD_MODE_TMZ || base->precision != FDTD_PREC_FP32)
    return bfail (b, FDTD_ERR_UNSUPPORTED, "batches are 2-D TMz, FP32");
  if (base->use_tfsf || base->use_metamaterials)
    return bfail (b, FDTD_ERR_UNSUPPORTED, "batches provide PML and a centred point source (no TF/SF, no Drude)");
  if (base->layout != 0 || base->double_material_precision || base->current_source_mask)
    return bfail (b, FDTD_ERR_UNSUPPORTED,
                  "batches use the E_CENTERED layout, cell-centred materials and no current source");
  if (count < 1 || !sizes)
    return bfail (b, FDTD_ERR_ARG, "empty batch");
  int ndev = 0;
  if (cudaGetDeviceCount (&ndev) != cudaSuccess || device < 0 || device >= ndev)
    return bfail (b, FDTD_ERR_CUDA, "no such CUDA device");
  b->device = device;
  b->base = *base;
  BCK (cudaSetDevice (device));
  BCK (cudaDeviceGetAttribute (&b->sm_count, cudaDevAttrMultiProcessorCount, device));
  int coop = 0;
  BCK (cudaDeviceGetAttribute (&coop, cudaDevAttrCooperativeLaunch, device));
  if (!coop)
    return bfail (b, FDTD_ERR_UNSUPPORTED, "device cannot launch cooperative kernels");
  BCK (cudaStreamCreateWithFlags (&b->stream, cudaStreamNonBlocking));
  BCK (cudaEventCreate (&b->ev0));
  BCK (cudaEventCreate (&b->ev1));
  b->geo.resize (count);
  b->inst.resize (count);
  const float identity[6] = {1.f, 0.f, 1.f, 1.f, 1.f, 1.f};   // ([1]: S, once it is known)
  b->tab_host.assign (identity, identity + 6);
  for (int i = 0; i < count; ++i)
  {
    fdtd_config c = *base;
    c.size[0] = sizes[2 * i];
    c.size[1] = sizes[2 * i + 1];
    c.size[2] = 1;
    c.point_source[0] = c.size[0] / 2;
    c.point_source[1] = c.size[1] / 2;
    c.point_source[2] = 0;
    c.point_source_mask &= 1 << FDTD_EZ;
    std::string e = build_geometry (c, b->geo[i]);
    if (!e.empty ())
      return bfail (b, FDTD_ERR_ARG, "instance " + std::to_string (i) + ": " + e);
    const Geometry &g = b->geo[i];
    InstDev &in = b->inst[i];
    std::memset (&in, 0, sizeof (in));
    in.off = b->cells;
    in.nx = g.n[0];
    in.ny = g.n[1];
    in.tab = (int) b->tab_host.size ();
    in.ps = c.point_source_mask ? 1 : 0;
    b->cells += (long long) in.nx * in.ny;
    const double S = kC * g.dt / g.dx;
    b->tab_host[1] = (float) S;
    // tables: Ez ca1(x) sq1(x) p5(y) q5(y); Hx g4p(x) g4m(x) ca1(y) sq1(y); Hy p5(x) q5(x) g4p(y) g4m(y)
    struct Spec
    {
      int comp, axis, kind;
    };
    static const Spec spec[12] = {{EZ, 0, 0}, {EZ, 0, 1}, {EZ, 1, 2}, {EZ, 1, 3}, {HX, 0, 4}, {HX, 0, 5},
                                  {HX, 1, 0}, {HX, 1, 1}, {HY, 0, 2}, {HY, 0, 3}, {HY, 1, 4}, {HY, 1, 5}};
    for (const Spec &sp : spec)
    {
      std::vector<double> sg = sigma_at (g, sp.comp, sp.axis);
      for (double sv : sg)
      {
        double r = sv * g.dt / (2 * kEps0);
        double v;
        switch (sp.kind)
        {
          case 0: v = (1 - r) / (1 + r); break;
          case 1: v = S / (1 + r); break;
          case 2: v = (1 - r) / (1 + r); break;
          case 3: v = 1 / (1 + r); break;
          case 4: v = 1 + r; break;
          default: v = 1 - r; break;
        }
        b->tab_host.push_back ((float) v);
      }
    }
    const int comps[3] = {EZ, HX, HY};
    for (int ci = 0; ci < 3; ++ci)
      for (int a = 0; a < 2; ++a)
      {
        std::vector<double> sg = sigma_at (g, comps[ci], a);
        int lo = 0, hi = g.n[a];
        if (base->use_pml)
        {
          while (lo < g.n[a] && sg[lo] != 0.0)
            ++lo;
          hi = lo;
          while (hi < g.n[a] && sg[hi] == 0.0)
            ++hi;
        }
        in.ilo[ci][a] = lo;
        in.ihi[ci][a] = hi;
      }
  }
  size_t cells = (size_t) b->cells;
  for (int s = 0; s < 2; ++s)
  {
    BALLOC (b->ez[s], cells * sizeof (float));
    BALLOC (b->hx[s], cells * sizeof (float));
    BALLOC (b->hy[s], cells * sizeof (float));
    if (base->use_pml)
    {
      BALLOC (b->aez[s], cells * sizeof (float));
      BALLOC (b->ahx[s], cells * sizeof (float));
      BALLOC (b->ahy[s], cells * sizeof (float));
    }
  }
  BALLOC (b->eps, cells * sizeof (float));
  fdtdb::fill_float_kernel<<<b->sm_count * 8, 256, 0, b->stream>>> (b->eps, cells, 1.f);
  BALLOC (b->d_tab, b->tab_host.size () * sizeof (float));
  BCK (cudaMemcpyAsync (b->d_tab, b->tab_host.data (), b->tab_host.size () * sizeof (float), cudaMemcpyHostToDevice,
                        b->stream));
  // per instance, each buffer set as the current one
  std::vector<Tile2D> dev (b->inst.size ());
  for (int set = 0; set < 2; ++set)
  {
    for (size_t i = 0; i < b->inst.size (); ++i)
    {
      const InstDev &in = b->inst[i];
      Tile2D &t = dev[i];
      std::memset (&t, 0, sizeof (t));
      t.nu = in.nx;
      t.nv = in.ny;
      t.use_pml = base->use_pml;
      t.courant = (float) (kC * b->geo[i].dt / b->geo[i].dx);
      t.scale[0] = 1.f;
      t.scale[1] = (float) kEta0B;
      t.pu = in.nx / 2;
      t.pv = in.ny / 2;
      t.src_row = 1;
      const float *T = b->d_tab + in.tab, *I = b->d_tab;
      const int nx = in.nx, ny = in.ny;
      const float *ez[4] = {T, T + nx, T + 2 * nx, T + 2 * nx + ny};
      T += 2 * nx + 2 * ny;
      const float *hx[4] = {T, T + nx, T + 2 * nx, T + 2 * nx + ny};
      T += 2 * nx + 2 * ny;
      const float *hy[4] = {T, T + nx, T + 2 * nx, T + 2 * nx + ny};
      const float *tab[3][6] = {{ez[0], ez[1], ez[2], ez[3], I + 4, I + 5},
                                {hx[2], hx[3], I + 2, I + 3, hx[0], hx[1]},
                                {I + 0, I + 1, hy[0], hy[1], hy[2], hy[3]}};
      float *const f[3][2] = {{b->ez[0], b->ez[1]}, {b->hx[0], b->hx[1]}, {b->hy[0], b->hy[1]}};
      float *const x[3][2] = {{b->aez[0], b->aez[1]}, {b->ahx[0], b->ahx[1]}, {b->ahy[0], b->ahy[1]}};
      for (int j = 0; j < 3; ++j)
      {
        TileComp &c = t.comp[j];
        c.nmat = 1;
        c.mat = j == 0 ? b->eps + in.off : nullptr;
        c.in = f[j][set] + in.off;
        c.out = f[j][1 - set] + in.off;
        if (base->use_pml)
        {
          c.aux_in = x[j][set] + in.off;
          c.aux_out = x[j][1 - set] + in.off;
        }
        for (int q = 0; q < 6; ++q)
          c.tab[q] = tab[j][q];
        for (int a = 0; a < 2; ++a)
        {
          c.ilo[a] = in.ilo[j][a];
          c.ihi[a] = in.ihi[j][a];
        }
        c.source = j == 0 && in.ps;
      }
    }
    BALLOC (b->d_inst[set], dev.size () * sizeof (Tile2D));
    BCK (cudaMemcpyAsync (b->d_inst[set], dev.data (), dev.size () * sizeof (Tile2D), cudaMemcpyHostToDevice,
                          b->stream));
    BCK (cudaStreamSynchronize (b->stream));
  }
  std::vector<PatchDev> patches;
  for (int i = 0; i < count; ++i)
    for (int u = 1; u <= b->inst[i].nx - 2; u += kCellRows)
      for (int v = 1; v <= b->inst[i].ny - 2; v += kCellCols)
        patches.push_back ({i, u, v});
  b->npatches = (int) patches.size ();
  BALLOC (b->d_geo, b->inst.size () * sizeof (InstDev));
  BCK (cudaMemcpyAsync (b->d_geo, b->inst.data (), b->inst.size () * sizeof (InstDev), cudaMemcpyHostToDevice,
                        b->stream));
  BALLOC (b->d_patches, patches.size () * sizeof (PatchDev));
  BCK (cudaMemcpyAsync (b->d_patches, patches.data (), patches.size () * sizeof (PatchDev), cudaMemcpyHostToDevice,
                        b->stream));
  BALLOC (b->d_counters, 4 * sizeof (unsigned));
  BALLOC (b->d_generation, sizeof (unsigned));
  BALLOC (b->d_err, sizeof (int));
  BCK (cudaStreamSynchronize (b->stream));
  return build_tiles (b, b->x_chunk);
}

int ensure_src (fdtd_batch *b, size_t n)
{
  BCK (cudaStreamSynchronize (b->stream));   // the previous launch may still read the pinned table
  if (n <= b->src_cap)
    return FDTD_OK;
  if (b->h_src)
    cudaFreeHost (b->h_src);
  b->h_src = nullptr;
  if (b->d_src)
  {
    auto it = std::find (b->allocs.begin (), b->allocs.end (), (void *) b->d_src);
    if (it != b->allocs.end ())
      b->allocs.erase (it);
    cudaFree (b->d_src);
    b->d_src = nullptr;
  }
  size_t cap = std::max<size_t> (n, 1024);
  BALLOC (b->d_src, (cap + 1) * sizeof (double));
  BCK (fdtdb::pinned_malloc ((void **) &b->h_src, cap * sizeof (double)));
  b->src_cap = cap;
  drop_graph (b);
  return FDTD_OK;
}

// One call = one persistent launch; captured into a CUDA graph (source
// upload, counter reset, kernel) unless capture is refused, in which case
// the same three operations are issued directly.
int step_batch (fdtd_batch *b, uint32_t t_start, uint32_t n, bool allow_graph)
{
  int r = ensure_src (b, n);
  if (r != FDTD_OK)
    return r;
  for (uint32_t s = 0; s < n; ++s)
    b->h_src[s] = fdtdb::point_source (b->geo[0], t_start + s, false);
  BCK (cudaEventRecord (b->ev0, b->stream));
  bool launched = false;
  if (allow_graph && b->use_graph)
  {
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture (b->stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess)
    {
      int er = enqueue (b, t_start, n);
      cudaError_t ee = cudaStreamEndCapture (b->stream, &g);
      if (er == FDTD_OK && ee == cudaSuccess && g)
      {
        cudaError_t ie;
        if (b->graph)
        {
          cudaGraphExecUpdateResultInfo info;
          ie = cudaGraphExecUpdate (b->graph, g, &info);
          if (ie != cudaSuccess)
          {
            cudaGetLastError ();
            drop_graph (b);
          }
        }
        if (!b->graph)
          ie = cudaGraphInstantiate (&b->graph, g, 0);
        if (ie == cudaSuccess && cudaGraphLaunch (b->graph, b->stream) == cudaSuccess)
        {
          launched = true;
          b->graph_ok = true;
        }
      }
      if (g)
        cudaGraphDestroy (g);
      if (!launched)
      {
        cudaGetLastError ();
        drop_graph (b);
        b->use_graph = false;
        b->graph_ok = false;
      }
    }
    else
    {
      cudaGetLastError ();
      b->use_graph = false;
    }
  }
  if (!launched)
  {
    r = enqueue (b, t_start, n);
    if (r != FDTD_OK)
      return r;
  }
  BCK (cudaEventRecord (b->ev1, b->stream));
  if (batch_rounds (b, t_start, n) & 1u)
    b->cur ^= 1;
  return FDTD_OK;
}

}  // namespace

extern "C" {

int fdtd_batch_create (const fdtd_config *base, int count, const int *sizes, int device, fdtd_batch **out)
{
  if (!base || !out)
    return FDTD_ERR_ARG;
  *out = nullptr;
  fdtd_batch *b = new (std::nothrow) fdtd_batch ();
  if (!b)
    return FDTD_ERR_NOMEM;
  int r = create_batch (b, base, count, sizes, device);
  if (r != FDTD_OK)
  {
    fdtd_batch_destroy (b);
    return r;
  }
  *out = b;
  return FDTD_OK;
}

int fdtd_batch_upload_eps (fdtd_batch *b, int instance, const double *host)
{
  if (!b || !host || instance < 0 || instance >= (int) b->inst.size ())
    return FDTD_ERR_ARG;
  BCK (cudaSetDevice (b->device));
  const fdtdb::InstDev &in = b->inst[instance];
  size_t n = (size_t) in.nx * in.ny;
  std::vector<float> f (n);
  for (size_t i = 0; i < n; ++i)
    f[i] = (float) host[i];
  BCK (cudaMemcpyAsync (b->eps + in.off, f.data (), n * sizeof (float), cudaMemcpyHostToDevice, b->stream));
  BCK (cudaStreamSynchronize (b->stream));
  return FDTD_OK;
}

int fdtd_batch_step (fdtd_batch *b, uint32_t t_start, uint32_t n_steps)
{
  if (!b)
    return FDTD_ERR_ARG;
  if (n_steps == 0)
    return FDTD_OK;
  BCK (cudaSetDevice (b->device));
  return step_batch (b, t_start, n_steps, true);
}

int fdtd_batch_sync (fdtd_batch *b, int64_t timeout_ns)
{
  if (!b)
    return FDTD_ERR_ARG;
  BCK (cudaSetDevice (b->device));
  if (timeout_ns < 0)
  {
    BCK (cudaStreamSynchronize (b->stream));
  }
  else
  {
    auto t0 = std::chrono::steady_clock::now ();
    for (;;)
    {
      cudaError_t e = cudaStreamQuery (b->stream);
      if (e == cudaSuccess)
        break;
      if (e != cudaErrorNotReady)
        return bfail (b, FDTD_ERR_CUDA, cudaGetErrorString (e));
      if (std::chrono::duration_cast<std::chrono::nanoseconds> (std::chrono::steady_clock::now () - t0).count ()
          >= timeout_ns)
        return bfail (b, FDTD_ERR_TIMEOUT, "sync timed out");
    }
  }
  float ms = 0.f;
  if (cudaEventElapsedTime (&ms, b->ev0, b->ev1) == cudaSuccess)
    b->last_ms = ms;
  int flag = 0;
  BCK (cudaMemcpy (&flag, b->d_err, sizeof (int), cudaMemcpyDeviceToHost));
  if (flag)
    return bfail (b, FDTD_ERR_DEVICE, "a grid barrier timed out");
  return FDTD_OK;
}

int fdtd_batch_download (fdtd_batch *b, int instance, int component, double *host)
{
  if (!b || !host || instance < 0 || instance >= (int) b->inst.size ()
      || (component != FDTD_EZ && component != FDTD_HX && component != FDTD_HY))
    return FDTD_ERR_ARG;
  int r = fdtd_batch_sync (b, -1);
  if (r != FDTD_OK)
    return r;
  const fdtdb::InstDev &in = b->inst[instance];
  size_t n = (size_t) in.nx * in.ny;
  const float *src = component == FDTD_EZ ? b->ez[b->cur] : (component == FDTD_HX ? b->hx[b->cur] : b->hy[b->cur]);
  // widened on the device a piece of rows at a time (an instance may have more
  // than 2^31 cells, and a batch that fills the device has no room for a second
  // copy of its largest one), each copied into the caller's buffer
  if (!b->stage)
  {
    size_t most = 0;
    for (const fdtdb::InstDev &i : b->inst)
      most = std::max (most, (size_t) i.nx * i.ny);
    most = std::min (most, kStageCells);
    BALLOC (b->stage, most * sizeof (double));
    b->stage_cells = most;
  }
  const double scale = component == FDTD_EZ ? 1.0 : 1.0 / fdtdb::kEta0B;
  // (whole groups of four rows keep every piece on a 16-byte boundary)
  const size_t fit = b->stage_cells / in.ny, piece = (fit >= 4 ? fit / 4 * 4 : fit) * in.ny;
  for (size_t at = 0; at < n; at += piece)
  {
    const size_t m = std::min (piece, n - at);
    fdtdb::launch_convert_out (b->stage, src + in.off + at, 1, m / in.ny, in.ny, in.ny, scale, b->stream);
    BCK (cudaGetLastError ());
    BCK (cudaMemcpyAsync (host + at, b->stage, m * sizeof (double), cudaMemcpyDeviceToHost, b->stream));
  }
  BCK (cudaStreamSynchronize (b->stream));
  return FDTD_OK;
}

int fdtd_batch_tune (fdtd_batch *b, int steps, int *choice)
{
  if (!b || steps < 1)
    return FDTD_ERR_ARG;
  BCK (cudaSetDevice (b->device));
  static const int tiles[] = {32, 64};
  static const int per_sm[] = {1, 2, 4};
  double best = 1e30;
  int bc = b->x_chunk, bs = b->ctas_per_sm;
  for (int c : tiles)
  {
    int r = build_tiles (b, c);
    if (r != FDTD_OK)
      return r;
    for (int s : per_sm)
    {
      if (s > max_ctas (c))
        continue;
      b->ctas_per_sm = s;
      b->tuning = true;
      r = step_batch (b, 1, (uint32_t) steps, false);
      b->tuning = false;
      if (r != FDTD_OK)
        return r;
      BCK (cudaStreamSynchronize (b->stream));
      float ms = 0.f;
      BCK (cudaEventElapsedTime (&ms, b->ev0, b->ev1));
      int flag = 0;
      BCK (cudaMemcpy (&flag, b->d_err, sizeof (int), cudaMemcpyDeviceToHost));
      if (flag)
        return bfail (b, FDTD_ERR_DEVICE, "a grid barrier timed out while tuning");
      if (ms < best)
      {
        best = ms;
        bc = c;
        bs = s;
      }
    }
  }
  // back to the state before tuning: zero fields and auxiliaries, t = 0
  size_t bytes = (size_t) b->cells * sizeof (float);
  for (int s = 0; s < 2; ++s)
  {
    float *arr[6] = {b->ez[s], b->hx[s], b->hy[s], b->aez[s], b->ahx[s], b->ahy[s]};
    for (float *a : arr)
      if (a)
        BCK (cudaMemsetAsync (a, 0, bytes, b->stream));
  }
  b->cur = 0;
  b->ctas_per_sm = bs;
  int r = build_tiles (b, bc);
  if (r != FDTD_OK)
    return r;
  drop_graph (b);
  b->use_graph = true;
  if (choice)
  {
    choice[0] = bc;
    choice[1] = fdtdb::kTileWarps;
    choice[2] = bs;
  }
  return FDTD_OK;
}

int fdtd_batch_info (const fdtd_batch *b, int64_t *cells, int *graph_used, double *last_ms)
{
  if (!b)
    return FDTD_ERR_ARG;
  if (cells)
    *cells = b->cells;
  if (graph_used)
    *graph_used = b->graph_ok ? 1 : 0;
  if (last_ms)
    *last_ms = b->last_ms;
  return FDTD_OK;
}

void fdtd_batch_destroy (fdtd_batch *b)
{
  if (!b)
    return;
  cudaSetDevice (b->device);
  if (b->stream)
    cudaStreamSynchronize (b->stream);
  drop_graph (b);
  for (void *p : b->allocs)
    cudaFree (p);
  if (b->h_src)
    cudaFreeHost (b->h_src);
  if (b->ev0)
    cudaEventDestroy (b->ev0);
  if (b->ev1)
    cudaEventDestroy (b->ev1);
  if (b->stream)
    cudaStreamDestroy (b->stream);
  delete b;
}

int fdtd_batch_set_wait_limit (fdtd_batch *b, int64_t limit_ns)
{
  if (!b)
    return FDTD_ERR_ARG;
  b->wait_limit_ns = limit_ns > 0 ? limit_ns : 0;
  return FDTD_OK;
}

const char *fdtd_batch_last_error (const fdtd_batch *b)
{
  return b ? b->err.c_str () : "";
}

}  // extern "C"
