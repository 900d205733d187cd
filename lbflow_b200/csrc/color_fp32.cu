// Two-phase step, FP32 storage.
#include "color_step.cuh"

namespace lbf {

void launch_color_fp32(int dims, int collision, bool pull, int out, const ColorLaunch& a)
{
    if (dims == 3) dispatch_coll<D3Q19, StoreF32Full>(collision, pull, out, a);
    else dispatch_coll<D2Q9, StoreF32Full>(collision, pull, out, a);
}

}  // namespace lbf
