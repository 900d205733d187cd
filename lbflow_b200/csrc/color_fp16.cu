// Two-phase step, FP16 storage.
#include "color_step.cuh"

namespace lbf {

void launch_color_fp16(int dims, int collision, bool pull, int out, const ColorLaunch& a)
{
    if (dims == 3) dispatch_coll<D3Q19, ColorPacked<D3Q19, __half>>(collision, pull, out, a);
    else dispatch_coll<D2Q9, ColorPacked<D2Q9, __half>>(collision, pull, out, a);
}

}  // namespace lbf
