// Two-phase step, FP64 storage.
#include "color_step.cuh"

namespace lbf {

void launch_color_fp64(int dims, int collision, bool pull, int out, const ColorLaunch& a)
{
    if (dims == 3) dispatch_coll<D3Q19, StoreF64>(collision, pull, out, a);
    else dispatch_coll<D2Q9, StoreF64>(collision, pull, out, a);
}

}  // namespace lbf
