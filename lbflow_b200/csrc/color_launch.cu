// Dispatch of the two-phase kernels by storage type.
#include "internal.h"
#include "../../include/lbflow.h"

namespace lbf {

void launch_color_fp64(int dims, int collision, bool pull, int out, const ColorLaunch& a);
void launch_color_fp32(int dims, int collision, bool pull, int out, const ColorLaunch& a);
void launch_color_fp16(int dims, int collision, bool pull, int out, const ColorLaunch& a);
void launch_color_bf16(int dims, int collision, bool pull, int out, const ColorLaunch& a);

void launch_color(int dims, int storage, int collision, bool pull, int out, const ColorLaunch& a)
{
    // The two-phase path stores full populations (FP64, or FP32 at reduced
    // precision), or the total and the component-0 share in 16 bits each.
    switch (storage) {
    case LBF_STORE_FP64: launch_color_fp64(dims, collision, pull, out, a); break;
    case LBF_STORE_FP16: launch_color_fp16(dims, collision, pull, out, a); break;
    case LBF_STORE_BF16: launch_color_bf16(dims, collision, pull, out, a); break;
    default: launch_color_fp32(dims, collision, pull, out, a); break;
    }
}

void launch_color_init(int dims, int storage, const Grid& g, const Force& F, const ColorParams& P,
                       const uint8_t* phase, void* f, cudaStream_t s)
{
    const unsigned threads = 256, blocks = blocks_for(g.nf, threads);
    if (blocks == 0) return;
    uint16_t* h = static_cast<uint16_t*>(f);
    if (dims == 3) {
        if (storage == LBF_STORE_FP64) color_init<D3Q19, StoreF64><<<blocks, threads, 0, s>>>(g, F, P, phase, (double*)f);
        else if (storage == LBF_STORE_FP16)
            color_init<D3Q19, ColorPacked<D3Q19, __half>><<<blocks, threads, 0, s>>>(g, F, P, phase, h);
        else if (storage == LBF_STORE_BF16)
            color_init<D3Q19, ColorPacked<D3Q19, __nv_bfloat16>><<<blocks, threads, 0, s>>>(g, F, P, phase, h);
        else color_init<D3Q19, StoreF32Full><<<blocks, threads, 0, s>>>(g, F, P, phase, (float*)f);
    } else {
        if (storage == LBF_STORE_FP64) color_init<D2Q9, StoreF64><<<blocks, threads, 0, s>>>(g, F, P, phase, (double*)f);
        else if (storage == LBF_STORE_FP16)
            color_init<D2Q9, ColorPacked<D2Q9, __half>><<<blocks, threads, 0, s>>>(g, F, P, phase, h);
        else if (storage == LBF_STORE_BF16)
            color_init<D2Q9, ColorPacked<D2Q9, __nv_bfloat16>><<<blocks, threads, 0, s>>>(g, F, P, phase, h);
        else color_init<D2Q9, StoreF32Full><<<blocks, threads, 0, s>>>(g, F, P, phase, (float*)f);
    }
}

}  // namespace lbf
