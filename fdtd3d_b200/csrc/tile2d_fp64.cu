// tile2d_fp64.cu - the FP64 plain form's 2-D tile kernel (--fmad=false).
#include "tile2d.cuh"

namespace fdtdb {

// 32 x 32 tiles while they fit the SMs once (18 x 18 own cells), else 64 x 32
// (50 x 18 own).
int launch_tile2d_fp64 (const Tile2D &p, int sm_count, cudaStream_t s)
{
  if (tile2d_count (p, 2, 1) <= sm_count)
    return tile2d_launch<double, double, 2, 1> (p, s);
  return tile2d_launch<double, double, 4, 1> (p, s);
}

}  // namespace fdtdb
