// Template instantiation and dispatch of the single-phase kernels.
#include "internal.h"
#include "../../include/lbflow.h"

namespace lbf {

namespace {
// Which steps take their sources from the table: 16-bit storage (see Links).
template <class L, class S> struct UseLinks {
    static constexpr bool value = L::D == 3 && sizeof(typename S::T) == 2;
};

// Whether the step's launch updates the nb boundary nodes too; otherwise a launch
// of their own follows it.  Inside, their chain overlaps with the other nodes'
// work, but FP64 then runs the whole step at five blocks per SM instead of seven,
// and a boundary node's populations, written apart from their neighbours', leave
// sectors that large geometries write back and read in parts.  Inside / apart, us
// per step (nodes, boundary nodes):
//   FP64  537 k, 21 k 37.6 / 42.2;  482 k, 44 k 41.5 / 43.7;  865 k, 8 k 52.4 /
//         54.0;  894 k, 19 k 60.6 / 60.5;  671 k, 78 k 70.6 / 65.9;  1.73 M, 8 k
//         103 / 96;  2.5 M, 78 k 199 / 174;  5.1 M, 129 k 396 / 341
//   FP32  537 k, 21 k 18.7 / 23.5;  1.05 M, 44 k 47.9 / 49.7;  2.9 M, 19 k 99.0 /
//         102.4;  783 k, 178 k 44.5 / 45.6;  1.52 M, 56 k 74.5 / 72.2;  2.5 M, 78 k
//         125 / 117;  5.1 M, 129 k 247 / 228;  10 M, 28 k 321 / 309
//   FP16  537 k, 21 k 15.3 / 27.1;  5.1 M, 129 k 189 / 227;  3.5 M, 317 k 148 / 188
template <class S> bool zou_he_inside(uint64_t nf, uint64_t nb)
{
    if constexpr (sizeof(typename S::T) == 8) return nf + 8 * nb <= 950000;
    if constexpr (sizeof(typename S::T) == 4) return nf * nb <= 80000000000ull;
    return true;
}

template <class L, class S>
void dispatch(bool mrt, bool pull, int out, const ScspLaunch& a)
{
    using T = typename S::T;
    const T* fin = static_cast<const T*>(a.fin);
    T* fout = static_cast<T*>(a.fout);
    const unsigned threads = 128, blocks = blocks_for(a.g.nf, threads);
    if (blocks == 0) return;
    (void)mrt;   // the collision rates (SRT or MRT) are in a.P.rate
    // At t = 0 (no pull) the boundary nodes hold rho0 at rest, which the
    // ordinary update reproduces from their initial populations.
    const unsigned zall = pull ? blocks_for(a.zh.n, threads) : 0;
    const unsigned zb = zou_he_inside<S>(a.g.nf, a.zh.n) ? zall : 0;
    auto step = [&](auto kernel) {
        launch_pdl(kernel, zb + blocks, threads, a.stream, a.g, a.F, a.P, fin, fout, a.mo, out, a.err, a.ein, a.eout,
                   a.zh, zb, a.links);
    };
    if (!pull) {
        scsp_step<L, S, false, false, false><<<blocks, threads, 0, a.stream>>>(
            a.g, a.F, a.P, fin, fout, a.mo, out, a.err, a.ein, a.eout, a.zh, 0u, a.links);
        return;
    }
    bool done = false;
    if constexpr (UseLinks<L, S>::value) {
        if (a.links.row) {
            if (zb) step(scsp_step<L, S, true, true, true>);
            else step(scsp_step<L, S, true, false, true>);
            done = true;
        }
    }
    if (!done) {
        if (zb) step(scsp_step<L, S, true, true, false>);
        else step(scsp_step<L, S, true, false, false>);
    }
    if constexpr (sizeof(T) >= 4)
        if (zall && !zb)
            launch_pdl(scsp_zou_he_pass<L, S>, zall, threads, a.stream, a.g, a.P, a.zh, fin, fout, a.mo, a.out, a.err,
                       a.ein, a.eout);
}

template <class L>
void dispatch_storage(int storage, bool mrt, bool pull, int out, const ScspLaunch& a)
{
    switch (storage) {
    case LBF_STORE_FP64: dispatch<L, StoreF64>(mrt, pull, out, a); break;
    case LBF_STORE_FP16: dispatch<L, StoreF16<L>>(mrt, pull, out, a); break;
    case LBF_STORE_BF16: dispatch<L, StoreBF16<L>>(mrt, pull, out, a); break;
    case LBF_STORE_BFP16: dispatch<L, StoreBFP16<L>>(mrt, pull, out, a); break;
    default: dispatch<L, StoreF32<L>>(mrt, pull, out, a); break;
    }
}

// The resident kernel's launch (nodes = nullptr), or the number of nodes the
// device holds at once.
template <class L, class S>
cudaError_t resident(const ScspLaunch* a, const Resident* r, uint32_t* nodes)
{
    using T = typename S::T;
    constexpr unsigned threads = kResidentThreads;
    if (nodes) {
        int dev = 0, sms = 0, per = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, scsp_resident<L, S>, threads, 0);
        *nodes = (uint32_t)(sms * per) * threads;
        return e;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks_for(a->g.nf, threads));
    cfg.blockDim = dim3(threads);
    cfg.stream = a->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, scsp_resident<L, S>, a->g, a->F, a->P, static_cast<const T*>(a->fin),
                              static_cast<T*>(a->fout), *r, a->mo, a->out, a->err);
}

template <class L>
cudaError_t resident_storage(int storage, const ScspLaunch* a, const Resident* r, uint32_t* nodes)
{
    switch (storage) {
    case LBF_STORE_FP64: return resident<L, StoreF64>(a, r, nodes);
    case LBF_STORE_FP32: return resident<L, StoreF32<L>>(a, r, nodes);
    case LBF_STORE_FP16: return resident<L, StoreF16<L>>(a, r, nodes);
    case LBF_STORE_BF16: return resident<L, StoreBF16<L>>(a, r, nodes);
    default: return cudaErrorNotSupported;
    }
}

template <class L>
void init_storage(int storage, const Grid& g, const Force& F, double rho0, void* f, int8_t* e, cudaStream_t s)
{
    const unsigned threads = 256, blocks = blocks_for(g.nf, threads);
    if (blocks == 0) return;
    switch (storage) {
    case LBF_STORE_FP64: scsp_init<L, StoreF64><<<blocks, threads, 0, s>>>(g, F, rho0, (double*)f, e); break;
    case LBF_STORE_FP16: scsp_init<L, StoreF16<L>><<<blocks, threads, 0, s>>>(g, F, rho0, (__half*)f, e); break;
    case LBF_STORE_BF16: scsp_init<L, StoreBF16<L>><<<blocks, threads, 0, s>>>(g, F, rho0, (__nv_bfloat16*)f, e); break;
    case LBF_STORE_BFP16: scsp_init<L, StoreBFP16<L>><<<blocks, threads, 0, s>>>(g, F, rho0, (int16_t*)f, e); break;
    default: scsp_init<L, StoreF32<L>><<<blocks, threads, 0, s>>>(g, F, rho0, (float*)f, e); break;
    }
}
template <class L>
void init_eq_storage(int storage, const Grid& g, const Force& F, double rho0, const float* fields, uint32_t ld,
                     void* f, int8_t* e, cudaStream_t s)
{
    const unsigned threads = 256, blocks = blocks_for(g.nf, threads);
    if (blocks == 0) return;
    switch (storage) {
    case LBF_STORE_FP64: scsp_init_eq<L, StoreF64><<<blocks, threads, 0, s>>>(g, F, rho0, fields, ld, (double*)f, e); break;
    case LBF_STORE_FP16: scsp_init_eq<L, StoreF16<L>><<<blocks, threads, 0, s>>>(g, F, rho0, fields, ld, (__half*)f, e); break;
    case LBF_STORE_BF16: scsp_init_eq<L, StoreBF16<L>><<<blocks, threads, 0, s>>>(g, F, rho0, fields, ld, (__nv_bfloat16*)f, e); break;
    case LBF_STORE_BFP16: scsp_init_eq<L, StoreBFP16<L>><<<blocks, threads, 0, s>>>(g, F, rho0, fields, ld, (int16_t*)f, e); break;
    default: scsp_init_eq<L, StoreF32<L>><<<blocks, threads, 0, s>>>(g, F, rho0, fields, ld, (float*)f, e); break;
    }
}
template <class L>
void add_density_storage(int storage, const Grid& g, const float* drho, void* f, int8_t* e, double rho0,
                         cudaStream_t s)
{
    const unsigned threads = 256, blocks = blocks_for(g.nf, threads);
    if (blocks == 0) return;
    switch (storage) {
    case LBF_STORE_FP64: scsp_add_density<L, StoreF64><<<blocks, threads, 0, s>>>(g, drho, (double*)f, e, rho0); break;
    case LBF_STORE_FP16: scsp_add_density<L, StoreF16<L>><<<blocks, threads, 0, s>>>(g, drho, (__half*)f, e, rho0); break;
    case LBF_STORE_BF16: scsp_add_density<L, StoreBF16<L>><<<blocks, threads, 0, s>>>(g, drho, (__nv_bfloat16*)f, e, rho0); break;
    case LBF_STORE_BFP16: scsp_add_density<L, StoreBFP16<L>><<<blocks, threads, 0, s>>>(g, drho, (int16_t*)f, e, rho0); break;
    default: scsp_add_density<L, StoreF32<L>><<<blocks, threads, 0, s>>>(g, drho, (float*)f, e, rho0); break;
    }
}
}  // namespace

bool scsp_uses_links(int dims, int storage)
{
    return dims == 3 && storage != LBF_STORE_FP64 && storage != LBF_STORE_FP32;
}

void launch_build_links(const Grid& g, uint4* row, uint32_t* mask, uint4* base, cudaStream_t s)
{
    const unsigned blocks = blocks_for(g.nf, kLinkTile);
    if (blocks) build_links<D3Q19><<<blocks, kLinkTile, 0, s>>>(g, row, mask, base);
}

void launch_scsp_add_density(int dims, int storage, const Grid& g, const float* drho, void* f, int8_t* e,
                             double rho0, cudaStream_t s)
{
    if (dims == 3) add_density_storage<D3Q19>(storage, g, drho, f, e, rho0, s);
    else add_density_storage<D2Q9>(storage, g, drho, f, e, rho0, s);
}

void launch_scsp_init_eq(int dims, int storage, const Grid& g, const Force& F, double rho0, const float* fields,
                         uint32_t ld, void* f, int8_t* e, cudaStream_t s)
{
    if (dims == 3) init_eq_storage<D3Q19>(storage, g, F, rho0, fields, ld, f, e, s);
    else init_eq_storage<D2Q9>(storage, g, F, rho0, fields, ld, f, e, s);
}

void launch_scsp(int dims, int storage, bool mrt, bool pull, int out, const ScspLaunch& a)
{
    if (dims == 3) dispatch_storage<D3Q19>(storage, mrt, pull, out, a);
    else dispatch_storage<D2Q9>(storage, mrt, pull, out, a);
}

cudaError_t launch_scsp_resident(int dims, int storage, const ScspLaunch& a, const Resident& r)
{
    return dims == 3 ? resident_storage<D3Q19>(storage, &a, &r, nullptr) : resident_storage<D2Q9>(storage, &a, &r, nullptr);
}

cudaError_t scsp_resident_nodes(int dims, int storage, uint32_t* nodes)
{
    return dims == 3 ? resident_storage<D3Q19>(storage, nullptr, nullptr, nodes)
                     : resident_storage<D2Q9>(storage, nullptr, nullptr, nodes);
}

void launch_scsp_init(int dims, int storage, const Grid& g, const Force& F, double rho0,
                      void* f, int8_t* e, cudaStream_t s)
{
    if (dims == 3) init_storage<D3Q19>(storage, g, F, rho0, f, e, s);
    else init_storage<D2Q9>(storage, g, F, rho0, f, e, s);
}

}  // namespace lbf
