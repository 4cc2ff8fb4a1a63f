// tile2d_fast.cu - the FP32 and FP16-storage forms' 2-D tile kernel.
#include "tile2d.cuh"

namespace fdtdb {

namespace {

// 32 x 32 tiles while they fit the SMs once (18 x 18 own cells), else 64 x 64
// (50 x 50 own).
template <typename T>
int launch_t (const Tile2D &p, int sm_count, cudaStream_t s)
{
  if (tile2d_count (p, 2, 1) <= sm_count)
    return tile2d_launch<T, float, 2, 1> (p, s);
  return tile2d_launch<T, float, 4, 2> (p, s);
}

}  // namespace

int launch_tile2d_fast (const Tile2D &p, bool fp16, int sm_count, cudaStream_t s)
{
  return fp16 ? launch_t<__half> (p, sm_count, s) : launch_t<float> (p, sm_count, s);
}

}  // namespace fdtdb
