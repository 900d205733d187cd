// Internal interfaces between the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <utility>
#include "kernels.cuh"
#include "color.cuh"
#include "resident.cuh"

namespace lbf {

struct ScspLaunch {
    Grid g;
    Force F;
    ScspParams P;
    const void* fin;
    void* fout;
    Macros mo;
    uint32_t* err;
    cudaStream_t stream;
    const int8_t* ein;   // block exponents of fin (block-scaled storage only)
    int8_t* eout;
    int out;             // kOutMacros / kOutAdjacent of this step
    ZouHe zh;            // PB/VB boundary nodes (n = 0: none)
    Links links;         // table of pull sources (row = nullptr: none)
};

struct ColorLaunch {
    Grid g;
    Force F;
    ColorParams P;
    ColorWall W;
    const void* fin;   // [2][Q][nfp]
    void* fout;
    double2* dens;     // [nfp] component densities (rho0, rho1) of this step (written by pass 1)
    double* phid;      // [N] phase field (rho0 - rho1)/rho per voxel (solid voxels: kSolidPhi)
    Macros mo;
    uint32_t* err;
    cudaStream_t stream;
    ZouHe zh;          // PB/VB boundary nodes (n = 0: none)
    Film film;         // half-permeable film bitmaps (nullptr: none)
};

// storage: LBF_STORE_* value; dims: 2 or 3.
void launch_scsp(int dims, int storage, bool mrt, bool pull, int out, const ScspLaunch& a);
// The table of pull sources: whether a storage's steps use it, and its fill.
bool scsp_uses_links(int dims, int storage);
void launch_build_links(const Grid& g, uint4* row, uint32_t* mask, uint4* base, cudaStream_t s);
void launch_scsp_init(int dims, int storage, const Grid& g, const Force& F, double rho0,
                      void* f, int8_t* eout, cudaStream_t s);
// All steps of a call in one launch (resident.cuh): a.out applies to the last.
// The caller keeps nf within scsp_resident_nodes (0 where unsupported).
cudaError_t launch_scsp_resident(int dims, int storage, const ScspLaunch& a, const Resident& r);
cudaError_t scsp_resident_nodes(int dims, int storage, uint32_t* nodes);
void launch_scsp_add_density(int dims, int storage, const Grid& g, const float* drho, void* f, int8_t* eio,
                             double rho0, cudaStream_t s);
void launch_scsp_init_eq(int dims, int storage, const Grid& g, const Force& F, double rho0, const float* fields,
                         uint32_t ld, void* f, int8_t* eout, cudaStream_t s);
void launch_color(int dims, int storage, int collision, bool pull, int out, const ColorLaunch& a);
void launch_color_init(int dims, int storage, const Grid& g, const Force& F, const ColorParams& P,
                       const uint8_t* phase, void* f, cudaStream_t s);

// The library's stream-ordered device memory pool of a device (created on
// first use; keeps freed memory reserved for reuse up to a fixed amount), so
// that work repeated inside a run allocates without driver calls.
cudaError_t device_pool(int device, cudaMemPool_t* pool);

// Message returned by lbf_last_error(NULL) (calls without an engine).
void set_global_error(const std::string& msg);

// Launch with programmatic stream serialization: the kernel may start before
// the previous kernel of the stream has completed and calls pdl_wait() before
// it touches anything an earlier kernel writes or reads.
template <class... P, class... A>
void launch_pdl_shared(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t shared, cudaStream_t s,
                       A&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), unsigned blocks, unsigned threads, cudaStream_t s, A&&... args)
{
    launch_pdl_shared(kernel, blocks, threads, 0, s, std::forward<A>(args)...);
}

inline unsigned blocks_for(uint32_t n, unsigned threads) { return (n + threads - 1) / threads; }

}  // namespace lbf
