// Two-phase step, BF16 storage.
#include "color_step.cuh"

namespace lbf {

void launch_color_bf16(int dims, int collision, bool pull, int out, const ColorLaunch& a)
{
    if (dims == 3) dispatch_coll<D3Q19, ColorPacked<D3Q19, __nv_bfloat16>>(collision, pull, out, a);
    else dispatch_coll<D2Q9, ColorPacked<D2Q9, __nv_bfloat16>>(collision, pull, out, a);
}

}  // namespace lbf
