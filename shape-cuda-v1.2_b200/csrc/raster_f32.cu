// FP32 instantiation of the tile rasterizer (radar views of the batched FP32
// form: FP64 vertices, coverage and depths, FP32 shading and synthesis; FMA
// contraction allowed).
#include "raster_impl.cuh"

namespace shape {
void launch_raster_f32(const RasterArgs &a, cudaStream_t s) { launch_raster_t<float>(a, s); }
int raster_occupancy_f32(const RasterArgs &a) { return raster_occupancy_t<float>(a); }
cudaError_t configure_raster_f32() { return configure_raster_t<float>(); }
}  // namespace shape
