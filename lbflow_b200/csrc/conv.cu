// Implicit-GEMM 3D convolutions of the learned warm start on tcgen05 tensor
// cores (BF16 operands, FP32 accumulators in tensor memory).
//
// Two kernels cover every convolution of the operator and its gradients:
//
//  igemm  out[row][n] = act(sum_k A[row][k] W[n][k] + bias)
//         A is gathered on the fly from one or two channels-last sources
//         (periodic 3x3x3 taps, 2x2x2 stride-2 cells or single voxels), W is
//         a K-major weight matrix.  Epilogues: bf16 or fp32 rows, or a
//         scatter into the 8 fine voxels of each 2x2x2 cell (transposed
//         convolution and the data gradient of the strided one).
//         Forward convolutions and data gradients (flipped, transposed
//         weights) run here.
//  wgrad  out[i][j] = sum_row A[row][i] B[row][j], both operands MN-major
//         (channels contiguous), the long reduction over rows split across
//         CTAs with fixed-order partial sums.  Weight gradients run here.
//
// Block: 160 threads, warp-specialised.  Warps 0-3 (128 producer threads)
// gather 16-byte pieces with cp.async into a 2-stage ring of
// 128-byte-swizzled operand tiles; each producer's copies of a stage arrive
// on the stage's `full` mbarrier (cp.async.mbarrier.arrive, 128 arrivals), so
// no producer waits for its own loads.  One thread of warp 4 waits for
// `full`, issues four M=128 x N x K=16 MMAs per 64-wide K stage and commits
// them to the stage's `empty` mbarrier, which the producers wait on before
// refilling the slot; its last commit arrives on `done`.  The epilogue (warps
// 0-3) reads the accumulator rows back with tcgen05.ld (warp w owns TMEM
// lanes 32w..32w+31 = tile rows).  Every wait is bounded: on timeout the
// kernel sets LBF_ERR_MMA_TIMEOUT, stops issuing and still releases its
// tensor memory.
#include "../../include/lbflow.h"
#include "../../include/lbflow_operator.h"
#include "internal.h"
#include "umma.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

namespace {

using namespace lbf::umma;

constexpr int kProducers = 128;        // warps 0-3: operand gathers, then the epilogue
constexpr int kThreads = kProducers + 32;   // + warp 4: the MMA issuer
constexpr int kBM = 128;             // tile rows = UMMA M
constexpr int kBK = 64;              // K per stage: one 128-byte swizzle row of bf16
// Two stages: with the producers decoupled from the MMA issue, the number of
// CTAs an SM holds (set by shared memory: 4 at 49 KB each) matters more than
// the ring depth (measured on the heaviest launch: 2 stages 390 TFLOP/s,
// 3 stages 348, 4 stages 282, 5 stages 177).
constexpr int kStages = 2;
constexpr uint32_t kTileA = kBM * kBK * 2;
constexpr long long kWaitCycles = 4000000000LL;   // about 2 s at the boost clock

struct Gather {
    const uint16_t* src0;
    const uint16_t* src1;
    uint32_t c0, c1, ct;
    uint32_t in_d, in_h, in_w;
    uint32_t out_d, out_h, out_w;
    uint32_t ks, stride;
    int pad;
    uint32_t taps;
    uint32_t rows;
};

struct Coord {
    int b, z, y, x;   // GEMM-row voxel
};

__device__ __forceinline__ Coord row_coord(const Gather& g, uint32_t m) {
    Coord c;
    c.x = int(m % g.out_w);
    uint32_t t = m / g.out_w;
    c.y = int(t % g.out_h);
    t /= g.out_h;
    c.z = int(t % g.out_d);
    c.b = int(t / g.out_d);
    return c;
}

__device__ __forceinline__ int wrap(int v, int n) {
    return v < 0 ? v + n : (v >= n ? v - n : v);
}

__device__ __forceinline__ void tap_offsets(const Gather& g, uint32_t tap, int& dz, int& dy, int& dx) {
    const uint32_t k2 = g.ks * g.ks;
    dz = int(tap / k2);
    const uint32_t r = tap - uint32_t(dz) * k2;
    dy = int(r / g.ks);
    dx = int(r - uint32_t(dy) * g.ks);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

struct SmemRing {
    uint32_t a0, b0, b_bytes, full0, empty0, done, tmem_slot;
    __device__ uint32_t a(int s) const { return a0 + uint32_t(s) * kTileA; }
    __device__ uint32_t b(int s) const { return b0 + uint32_t(s) * b_bytes; }
    __device__ uint32_t full(int s) const { return full0 + uint32_t(s) * 8u; }
    __device__ uint32_t empty(int s) const { return empty0 + uint32_t(s) * 8u; }
};

__device__ __forceinline__ SmemRing carve(uint8_t* raw, uint32_t b_bytes) {
    SmemRing r;
    const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u;
    r.a0 = base;
    r.b0 = base + kStages * kTileA;
    r.b_bytes = b_bytes;
    r.full0 = r.b0 + kStages * b_bytes;
    r.empty0 = r.full0 + kStages * 8u;
    r.done = r.empty0 + kStages * 8u;
    r.tmem_slot = r.done + 8u;
    return r;
}

constexpr size_t smem_bytes(uint32_t b_bytes) {
    return 1024 + kStages * (kTileA + b_bytes) + (2 * kStages + 1) * 8 + 16;
}

// Allocation of `cols` TMEM columns by warp 0 and the barrier set-up.
__device__ __forceinline__ uint32_t prologue(const SmemRing& r, uint32_t cols) {
    if (threadIdx.x < 32) {
        tmem_alloc(r.tmem_slot, cols);
        tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(r.full(s), kProducers);
            mbar_init(r.empty(s), 1);
        }
        mbar_init(r.done, 1);
        mbar_init_fence();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    uint32_t t;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(t) : "r"(r.tmem_slot) : "memory");
    return t;
}

__device__ __forceinline__ void release(uint32_t tmem, uint32_t cols) {
    fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tmem_dealloc(tmem, cols);
}

// The shared producer / MMA pipeline.  Loader provides (producer threads)
//   load(chunk, stage)   cp.async the chunk's A and B tiles into the stage
//   adesc/bdesc(stage, kk)  descriptors of the kk-th K=16 slice
// Returns, in the producer threads, whether the accumulator is complete
// (every wait succeeded and `done` fired); false elsewhere or on a timeout.
template <class Loader>
__device__ bool mainloop(Loader& ld, const SmemRing& r, uint32_t nch, uint32_t tmem, uint32_t idesc) {
    const uint32_t warp = threadIdx.x >> 5;
    if (warp < uint32_t(kProducers / 32)) {
        bool ok = true;
        for (uint32_t c = 0; c < nch; ++c) {
            const int s = int(c % kStages);
            if (c >= uint32_t(kStages)) {
                // The slot's previous chunk must have been consumed by its MMAs.
                const bool w = mbar_wait(r.empty(s), ((c / kStages) - 1u) & 1u, kWaitCycles);
                ok = __all_sync(0xffffffffu, w);      // the warp leaves together (loads shuffle)
                if (!ok) break;
            }
            ld.load(c, s);
            cp_async_arrive(r.full(s));
        }
        cp_async_commit();          // wait_group only waits for committed copies
        cp_async_wait<0>();
        const bool d = mbar_wait(r.done, 0u, kWaitCycles);
        fence_after_sync();
        return ok && d;
    }
    if (threadIdx.x == uint32_t(kProducers)) {
        bool ok = true;
        for (uint32_t c = 0; c < nch; ++c) {
            const int s = int(c % kStages);
            ok = mbar_wait(r.full(s), (c / kStages) & 1u, kWaitCycles);
            if (!ok) break;
            // The producers' cp.async writes, made visible to the tensor
            // core's (async-proxy) reads of the stage.
            fence_async_shared();
            fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                mma_bf16(tmem, ld.adesc(s, kk), ld.bdesc(s, kk), idesc, (c | uint32_t(kk)) != 0u);
            commit(r.empty(s));
        }
        // `done` fires once every MMA issued above has completed (at once
        // when none was issued), also after a timeout, so the tensor memory
        // is never released under a running MMA.
        commit(r.done);
    }
    return false;
}

// ---------------------------------------------------------------- igemm ----

struct IgemmArgs {
    Gather g;
    const uint16_t* w;
    uint32_t n, k_pad;
    const float* bias;
    void* out;
    uint32_t mode, ld;
    uint32_t act;
    float slope;
    uint32_t* err;
};

// Voxel index of tap (dz, dy, dx) of row voxel c, and the address of channels
// [ch, ch + 8) of that voxel in whichever source holds them.
__device__ __forceinline__ size_t gather_vox(const Gather& g, const Coord& c, int dz, int dy, int dx) {
    const int z = wrap(int(g.stride) * c.z + dz - g.pad, int(g.in_d));
    const int y = wrap(int(g.stride) * c.y + dy - g.pad, int(g.in_h));
    const int x = wrap(int(g.stride) * c.x + dx - g.pad, int(g.in_w));
    return ((size_t(c.b) * g.in_d + z) * g.in_h + y) * g.in_w + x;
}
__device__ __forceinline__ const uint16_t* chan_ptr(const Gather& g, size_t vox, uint32_t ch) {
    return ch < g.c0 ? g.src0 + vox * g.c0 + ch : g.src1 + vox * g.c1 + (ch - g.c0);
}

// A tile: thread t owns tile row t and copies its 8 16-byte pieces of each
// 64-wide K stage.  When a stage lies inside one tap of one source (channel
// counts multiples of 64) the row's 128 bytes are contiguous in memory: one
// address per stage.  Otherwise the tap and channel advance piece by piece.
template <int BN>
struct IgemmLoader {
    const IgemmArgs& p;
    SmemRing r;
    Coord rc;
    bool rv;
    bool uniform;
    uint32_t n0;
    uint32_t sw;          // swizzle of the thread's row (row mod 8)
    uint32_t poff_b;      // swizzled byte offset of the thread's B piece
    // Uniform path: the K position of the next chunk (chunks come in order)
    // as tap (dz, dy, dx) and channel, advanced incrementally instead of by
    // divisions, and the row's unwrapped source origin stride * voxel - pad.
    uint32_t u_tap, u_ch;
    int u_dz, u_dy, u_dx;
    int oz, oy, ox;

    __device__ IgemmLoader(const IgemmArgs& a, const SmemRing& ring, uint32_t m0, uint32_t n0_)
        : p(a), r(ring), n0(n0_) {
        const uint32_t t = threadIdx.x;
        const uint32_t m = m0 + t;
        rv = m < p.g.rows;
        rc = row_coord(p.g, rv ? m : 0u);
        sw = t & 7u;
        poff_b = (((t & 7u) ^ ((t >> 3) & 7u)) << 4);
        uniform = (p.g.ct % kBK == 0) && (p.g.c1 == 0 || p.g.c0 % kBK == 0);
        u_tap = 0; u_ch = 0;
        u_dz = u_dy = u_dx = 0;
        oz = int(p.g.stride) * rc.z - p.g.pad;
        oy = int(p.g.stride) * rc.y - p.g.pad;
        ox = int(p.g.stride) * rc.x - p.g.pad;
    }

    __device__ void load(uint32_t chunk, int s) {
        const uint32_t t = threadIdx.x;
        const uint32_t a = r.a(s) + t * 128u;
        if (uniform) {
            // Each thread finds its row's 128 contiguous bytes; the copies are
            // then spread so that lanes 8q..8q+7 move the 8 pieces of one row
            // (coalesced), the row addresses passed by warp shuffles (a null
            // address marks a row past the end or a K position past the taps).
            const bool v = rv && u_tap < p.g.taps;
            const uint16_t* src = nullptr;
            if (v) {
                const int z = wrap(oz + u_dz, int(p.g.in_d));
                const int y = wrap(oy + u_dy, int(p.g.in_h));
                const int x = wrap(ox + u_dx, int(p.g.in_w));
                const size_t vox = ((size_t(rc.b) * p.g.in_d + z) * p.g.in_h + y) * p.g.in_w + x;
                src = chan_ptr(p.g, vox, u_ch);
            }
            // Next chunk: 64 channels further, carrying into the next tap.
            u_ch += kBK;
            if (u_ch >= p.g.ct) {
                u_ch = 0;
                ++u_tap;
                if (++u_dx == int(p.g.ks)) {
                    u_dx = 0;
                    if (++u_dy == int(p.g.ks)) { u_dy = 0; ++u_dz; }
                }
            }
            const uint32_t lane = t & 31u, wbase = t & ~31u, j = lane & 7u;
            const unsigned long long sp = reinterpret_cast<unsigned long long>(src);
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t rw = 4u * i + (lane >> 3);              // row within the warp
                const unsigned long long q = __shfl_sync(0xffffffffu, sp, int(rw));
                const uint32_t row = wbase + rw;
                const uint32_t dst = r.a(s) + row * 128u + ((j ^ (row & 7u)) << 4);
                cp_async16(dst, q ? reinterpret_cast<const uint16_t*>(q) + 8u * j : p.g.src0, q ? 16u : 0u);
            }
        } else {
            uint32_t k = chunk * kBK;
            uint32_t tap = k / p.g.ct;
            uint32_t ch = k - tap * p.g.ct;
            uint32_t cur = 0xffffffffu;
            size_t vox = 0;
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                const bool v = rv && tap < p.g.taps;
                if (v && tap != cur) {
                    int dz, dy, dx;
                    tap_offsets(p.g, tap, dz, dy, dx);
                    vox = gather_vox(p.g, rc, dz, dy, dx);
                    cur = tap;
                }
                cp_async16(a + ((j ^ sw) << 4), v ? chan_ptr(p.g, vox, ch) : p.g.src0, v ? 16u : 0u);
                ch += 8u;
                if (ch >= p.g.ct) { ch = 0; ++tap; }
            }
        }
        const uint32_t kb = chunk * kBK + (t & 7u) * 8u;
        const uint32_t b = r.b(s) + (t >> 3) * 128u + poff_b;
#pragma unroll
        for (int i = 0; i < BN / 16; ++i) {
            const uint32_t n = (t >> 3) + 16u * i;
            cp_async16(b + uint32_t(i) * 16u * 128u, p.w + size_t(n0 + n) * p.k_pad + kb, 16u);
        }
    }
    __device__ uint64_t adesc(int s, int kk) const { return desc_sw128(r.a(s) + 32u * kk, 16u, 1024u); }
    __device__ uint64_t bdesc(int s, int kk) const { return desc_sw128(r.b(s) + 32u * kk, 16u, 1024u); }
};

// Bias of 16 accumulator columns from nb, bias entries from `from` on, wrapping
// at p.ld in the scatter mode.  One branch for all 16: with one per column
// (bias or not, activation or not) these were the slowest part of the
// epilogue, 84 cycles a column.
__device__ __forceinline__ void add_bias(const IgemmArgs& p, float (&v)[16], uint32_t nb, uint32_t from) {
    if (!p.bias) return;
    const uint32_t period = p.mode == LBF_OUT_SCATTER2_BF16 ? p.ld : 0xffffffffu;
    float b[16];
#pragma unroll
    for (uint32_t e = 0; e < 16u; ++e) {
        b[e] = nb + e < p.n ? __ldg(p.bias + from) : 0.f;
        from = from + 1u == period ? 0u : from + 1u;
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] += b[e];
}

__device__ __forceinline__ void st_shared16(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) igemm_kernel(const __grid_constant__ IgemmArgs p) {
    extern __shared__ uint8_t smem_raw[];
    constexpr uint32_t kCols = BN < 32 ? 32 : BN;
    const SmemRing r = carve(smem_raw, BN * 128u);
    const uint32_t tmem = prologue(r, kCols);
    const uint32_t m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;

    IgemmLoader<BN> ld(p, r, m0, n0);
    const bool ok = mainloop(ld, r, p.k_pad / kBK, tmem, idesc_bf16(kBM, BN, false, false));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= uint32_t(kProducers / 32)) {
        release(tmem, kCols);
        return;
    }
    if (!ok && threadIdx.x == 0) atomicOr(p.err, LBF_ERR_MMA_TIMEOUT);

    const uint32_t row = m0 + warp * 32 + lane;
    const bool rvalid = ok && row < p.g.rows;
    Coord rc = row_coord(p.g, rvalid ? row : 0u);
    const float slope = p.act ? p.slope : 1.f;
#pragma unroll 1
    for (int col0 = 0; col0 < BN; col0 += 16) {
        float v[16];
        tmem_ld16(tmem + ((warp * 32u) << 16) + uint32_t(col0), v);
        if (!rvalid) continue;
        const uint32_t nb = n0 + col0;
        add_bias(p, v, nb, p.mode == LBF_OUT_SCATTER2_BF16 ? nb % p.ld : nb);
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = v[e] > 0.f ? v[e] : v[e] * slope;
        if (p.mode == LBF_OUT_F32) {
            float* o = static_cast<float*>(p.out) + size_t(row) * p.ld;
            for (int e = 0; e < 16; ++e)
                if (nb + e < p.n) o[nb + e] = v[e];
            continue;
        }
        uint16_t* o;
        uint32_t c;
        bool vec;
        if (p.mode == LBF_OUT_BF16) {
            o = static_cast<uint16_t*>(p.out) + size_t(row) * p.ld;
            c = nb;
            vec = (p.ld % 8u == 0u) && nb + 16 <= p.n;
        } else {
            // Scatter: n = tap * ld + c into fine voxel 2 * row + tap.
            const uint32_t tap = nb / p.ld;
            c = nb - tap * p.ld;
            const int dz = int(tap >> 2), dy = int((tap >> 1) & 1u), dx = int(tap & 1u);
            const size_t fd = 2u * p.g.out_d, fh = 2u * p.g.out_h, fw = 2u * p.g.out_w;
            const size_t vox = ((size_t(rc.b) * fd + 2 * rc.z + dz) * fh + 2 * rc.y + dy) * fw + 2 * rc.x + dx;
            o = static_cast<uint16_t*>(p.out) + vox * p.ld;
            vec = (p.ld % 16u == 0u) && nb + 16 <= p.n;
            if (!vec) {
                for (int e = 0; e < 16; ++e) {
                    const uint32_t n = nb + e;
                    if (n >= p.n) break;
                    const uint32_t tp = n / p.ld, cc = n - tp * p.ld;
                    const int ez = int(tp >> 2), ey = int((tp >> 1) & 1u), ex = int(tp & 1u);
                    const size_t vx = ((size_t(rc.b) * fd + 2 * rc.z + ez) * fh + 2 * rc.y + ey) * fw +
                                      2 * rc.x + ex;
                    __nv_bfloat16 h = __float2bfloat16_rn(v[e]);
                    static_cast<uint16_t*>(p.out)[vx * p.ld + cc] = *reinterpret_cast<uint16_t*>(&h);
                }
                continue;
            }
        }
        if (vec) {
            uint4 q0, q1;
            q0.x = pack_bf16(v[0], v[1]);   q0.y = pack_bf16(v[2], v[3]);
            q0.z = pack_bf16(v[4], v[5]);   q0.w = pack_bf16(v[6], v[7]);
            q1.x = pack_bf16(v[8], v[9]);   q1.y = pack_bf16(v[10], v[11]);
            q1.z = pack_bf16(v[12], v[13]); q1.w = pack_bf16(v[14], v[15]);
            reinterpret_cast<uint4*>(o + c)[0] = q0;
            reinterpret_cast<uint4*>(o + c)[1] = q1;
        } else {
            for (int e = 0; e < 16; ++e) {
                if (nb + e >= p.n) break;
                __nv_bfloat16 h = __float2bfloat16_rn(v[e]);
                o[c + e] = *reinterpret_cast<uint16_t*>(&h);
            }
        }
    }
    release(tmem, kCols);
}

// ---------------------------------------------------------------- conv3 ----

// Periodic 3x3x3 convolution of up to 64 channels from a tile with halo in
// shared memory.  igemm gathers the 27 taps of a row separately, so every
// input voxel crosses from L2 27 times, and with fewer than 64 channels its
// producers spend their time on tap arithmetic.  Here a block computes
// 8 (x) x 16 (y) x kCZ (z) outputs: it copies the 10 x 18 x (kCZ + 2) input
// voxels once, as 16-byte pieces [8 channels][voxel], which is the unswizzled
// K-major operand layout: 8 voxels along x are a core matrix, the 16 rows
// along y follow at the tile's row pitch, and a tap is a start address
// (dz, dy, dx) voxels further on.  The weights [tap][8 channels][n] stay in
// shared memory where they are few, else they stream through a ring of `stages`
// slots of `per` taps (a slot per tap is bound by the latency of its refill);
// each is used by the kCZ z slices' accumulators.  The K order per output is
// igemm's (tap, then channel), 16 at a time, so the result is too, bit for bit:
// channel counts that are a multiple of 16, and 8, where a K step takes two
// taps, one in each half (the halves of an operand lie any distance apart; 8 ->
// 16 at 96^3 33 us, 45 with a half of zeros beside each tap).  Other counts
// split a tap's channels over K steps and stay with igemm.
//
// Measured, igemm -> here: 16 -> 16 channels at 96^3 238 -> 48 us, 8 -> 16 187
// -> 33, 32 -> 16 (two sources) 403 -> 102, 32 -> 32 at 48^3 63 -> 22, 32 + 32
// -> 64 at 2 x 48^3 213 -> 80.  Per 64-channel block of 52,000 cycles: 10,000 for the halo
// (cp.async at 14 bytes a cycle), 28,000 for 432 MMAs (N = 64, 65 cycles each;
// operand reads alone need 48), the rest weights and epilogue.  Narrow inputs
// need several resident blocks to overlap those phases: the registers are
// capped for as many as shared memory holds (16 -> 16 at the compiler's 95
// registers, two blocks, 60 us; three 51, four 48).  8 producer warps: 16 take
// 96 us for 16 -> 16, their registers cost a resident block.
constexpr int kCX = 8, kCY = 16, kCZ = 4;
constexpr int kHX = kCX + 2, kHY = kCY + 2, kHZ = kCZ + 2;
constexpr int kHalo = kHX * kHY * kHZ;
// Channel groups' planes are one piece longer than the tile: the copies of a
// voxel's consecutive groups then fall into different banks.
constexpr uint32_t kPlane = (kHalo + 1) * 16;
constexpr int kTapStages = 3;      // most slots
constexpr int kConvProducers = 256, kConvThreads = kConvProducers + 32;
constexpr uint32_t kMaxConvC = 64;
struct TapRing { uint32_t per, stages; };

// Taps held with G channel groups: a 28th of zero weights completes the last
// pair of a single group, whose operand half then reads kZeros bytes of zeros.
constexpr uint32_t conv_taps(uint32_t groups) { return groups == 1 ? 28 : 27; }
constexpr uint32_t kZeros = ((kCY - 1) * kHX + 8) * 16;

constexpr size_t conv3_smem(uint32_t groups, uint32_t bn, TapRing r) {
    return 128 + size_t(groups) * kPlane + size_t(r.per) * r.stages * groups * bn * 16 + (groups == 1 ? kZeros : 0) +
           (2 + 2 * kTapStages) * 8 + 16;
}

// The epilogue's bf16 rows: a warp's 32, each padded by 16 bytes.
constexpr uint32_t conv3_pitch(uint32_t bn) { return bn * 2 + 16; }
constexpr uint32_t conv3_stage_bytes(uint32_t bn) { return kConvProducers * conv3_pitch(bn); }

// G: 8-channel groups held (1, 2, 4 or 8; those past the input's channels are
// zeros).
template <int BN, int G>
__global__ void __launch_bounds__(kConvThreads, G <= 2 ? 4 : (G == 4 ? 2 : 1))
conv3_kernel(const __grid_constant__ IgemmArgs p, const uint32_t tx, const uint32_t ty, const uint32_t tz,
             const TapRing ring) {
    extern __shared__ uint8_t smem_raw[];
    constexpr uint32_t kCols = kCZ * BN;
    constexpr uint32_t tap_bytes = G * BN * 16u;
    const uint32_t a0 = (smem_u32(smem_raw) + 127u) & ~127u;
    const uint32_t w0 = a0 + G * kPlane;
    const uint32_t slot_bytes = ring.per * tap_bytes;
    const uint32_t zeros = w0 + ring.stages * slot_bytes;
    const uint32_t bar = (zeros + (G == 1 ? kZeros : 0u) + 7u) & ~7u;
    const uint32_t full_a = bar, done = bar + 8u, full0 = bar + 16u, empty0 = full0 + kTapStages * 8u;
    const uint32_t slot = empty0 + kTapStages * 8u;

    if (threadIdx.x < 32) {
        tmem_alloc(slot, kCols);
        tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        mbar_init(full_a, kConvProducers);
        mbar_init(done, 1);
        for (int s = 0; s < kTapStages; ++s) {
            mbar_init(full0 + 8u * s, kConvProducers);
            mbar_init(empty0 + 8u * s, 1);
        }
        mbar_init_fence();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    uint32_t tmem;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem) : "r"(slot) : "memory");
    tmem = __shfl_sync(0xffffffffu, tmem, 0);

    uint32_t t = blockIdx.x;
    const int x0 = int(t % tx) * kCX;
    t /= tx;
    const int y0 = int(t % ty) * kCY;
    t /= ty;
    const int z0 = int(t % tz) * kCZ;
    const uint32_t b = t / tz;
    const uint32_t n0 = blockIdx.y * BN;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    bool ok = true;
    if (warp < uint32_t(kConvProducers / 32)) {
        // A thread copies one group of the 10 voxels of a tile row at a time, the
        // threads of consecutive groups side by side; its x offsets are the same
        // in every row.  Voxels past the grid belong to no valid output: any
        // address will do.
        constexpr uint32_t kStep = kConvProducers / G;
        auto inside = [](int v, int n) {
            v = wrap(v, n);
            return v < n ? v : 0;
        };
        const uint32_t g8 = threadIdx.x % G, first = threadIdx.x / G, ch = g8 * 8u;
        const bool in = ch < p.g.ct;
        const uint32_t c = ch < p.g.c0 ? p.g.c0 : p.g.c1;
        const uint16_t* const src = !in ? p.g.src0 : (ch < p.g.c0 ? p.g.src0 + ch : p.g.src1 + (ch - p.g.c0));
        const uint32_t bytes = in ? 16u : 0u;
        uint32_t xo[kHX];
#pragma unroll
        for (int i = 0; i < kHX; ++i) xo[i] = in ? uint32_t(inside(x0 + i - 1, int(p.g.in_w))) * c : 0u;
        for (uint32_t r = first; r < kHY * kHZ; r += kStep) {
            const uint32_t hz = r / kHY, hy = r - hz * kHY;
            const int z = inside(z0 + int(hz) - 1, int(p.g.in_d)), y = inside(y0 + int(hy) - 1, int(p.g.in_h));
            const size_t vox = ((size_t(b) * p.g.in_d + z) * p.g.in_h + y) * p.g.in_w;
            const uint16_t* const row = in ? src + vox * c : src;
            const uint32_t dst = a0 + g8 * kPlane + r * (kHX * 16u);
#pragma unroll
            for (int i = 0; i < kHX; ++i) cp_async16(dst + i * 16u, row + xo[i], bytes);
        }
        if (G == 1 && threadIdx.x < kZeros / 16u) cp_async16(zeros + threadIdx.x * 16u, p.g.src0, 0u);
        cp_async_arrive(full_a);
        const uint16_t* const wp = in ? p.w + size_t(n0) * p.k_pad + ch : p.w;
        const uint32_t total = conv_taps(G) / ring.per;
        for (uint32_t st = 0; st < total; ++st) {
            const uint32_t s = st % ring.stages;
            if (st >= ring.stages) {
                const bool w = mbar_wait(empty0 + 8u * s, (st / ring.stages - 1u) & 1u, kWaitCycles);
                ok = __all_sync(0xffffffffu, w);
                if (!ok) break;
            }
            for (uint32_t q = first; q < ring.per * BN; q += kStep) {
                const uint32_t tap = q / BN, n = q % BN;
                const bool real = in && st * ring.per + tap < 27u;
                cp_async16(w0 + s * slot_bytes + tap * tap_bytes + (g8 * BN + n) * 16u,
                           real ? wp + n * p.k_pad + (st * ring.per + tap) * p.g.ct : p.w, real ? 16u : 0u);
            }
            cp_async_arrive(full0 + 8u * s);
        }
        cp_async_commit();
        cp_async_wait<0>();
        const bool d = mbar_wait(done, 0u, kWaitCycles);
        fence_after_sync();
        ok = ok && d;
    } else {
        // The whole warp, converged; one lane issues.
        const uint32_t leader = elect_one();
        constexpr uint32_t idesc = idesc_bf16(kBM, BN, false, false);
        bool go = __all_sync(0xffffffffu, mbar_wait(full_a, 0u, kWaitCycles));
        // Descriptors differ in their start address (16-byte units) only.
        const uint64_t ad0 = desc_plain(a0, kPlane, kHX * 16u);
        const uint64_t bd0 = desc_plain(w0, BN * 16u, 128u);
        for (uint32_t st = 0; st < conv_taps(G) / ring.per && go; ++st) {
            const uint32_t s = st % ring.stages;
            go = __all_sync(0xffffffffu, mbar_wait(full0 + 8u * s, (st / ring.stages) & 1u, kWaitCycles));
            if (!go) break;
            fence_async_shared();
            fence_after_sync();
            if constexpr (G == 1) {
                // Taps 2 j and 2 j + 1 in one K step, the distance between them as
                // the distance between the operand's K halves.
                auto voxel = [](uint32_t tap) { return (tap / 9u * kHY + tap / 3u % 3u) * kHX + tap % 3u; };
                const uint64_t plain = desc_plain(a0, 0u, kHX * 16u);
                for (uint32_t j = 0; j < conv_taps(G) / 2u; ++j) {
                    const uint32_t at = voxel(2u * j), bd = 2u * j * BN;
#pragma unroll
                    for (uint32_t z = 0; z < uint32_t(kCZ); ++z) {
                        const uint32_t from = at + z * (kHX * kHY);
                        const uint32_t apart = 2u * j + 1u < 27u ? voxel(2u * j + 1u) - at : (zeros - a0) / 16u - from;
                        mma_bf16_warp(leader, tmem + z * BN, plain + from + (uint64_t(apart) << 16), bd0 + bd, idesc, j != 0u);
                    }
                }
            } else {
                for (uint32_t j = 0; j < ring.per; ++j) {
                    const uint32_t tap = st * ring.per + j;
                    const uint32_t dz = tap / 9u, dy = tap / 3u - 3u * dz, dx = tap % 3u;
                    uint64_t ad = ad0 + (dz * kHY + dy) * kHX + dx;
                    uint64_t bd = bd0 + (s * slot_bytes + j * tap_bytes) / 16u;
                    for (uint32_t k = 0; k < uint32_t(G); k += 2, ad += 2 * kPlane / 16u, bd += 2 * BN)
#pragma unroll
                        for (uint32_t z = 0; z < uint32_t(kCZ); ++z)
                            mma_bf16_warp(leader, tmem + z * BN, ad + z * (kHX * kHY), bd, idesc, (tap | k) != 0u);
                }
            }
            commit_warp(leader, empty0 + 8u * s);
        }
        commit_warp(leader, done);
    }
    if (warp >= uint32_t(kConvProducers / 32)) {
        release(tmem, kCols);
        return;
    }
    if (!ok && threadIdx.x == 0) atomicOr(p.err, LBF_ERR_MMA_TIMEOUT);

    // Accumulator row 8 y + x of each z slice; warp w reads lanes 32 (w mod 4)
    // on, four warps every other slice.
    const uint32_t quarter = warp & 3u, m = quarter * 32u + lane;
    const uint32_t x = uint32_t(x0) + (m & 7u), y = uint32_t(y0) + (m >> 3);
    // Rows that allow 16-byte bf16 stores go through shared memory (the tile is
    // no longer read): lanes then store consecutive pieces of the 8 voxels of a
    // tile row, one run in memory.
    const bool vec = p.mode == LBF_OUT_BF16 && p.ld % 8u == 0u && p.n % 8u == 0u;
    const float slope = p.act ? p.slope : 1.f;
    constexpr uint32_t kPitch = conv3_pitch(BN), kParts = BN / 8u;
    const uint32_t stage = a0 + warp * 32u * kPitch;
#pragma unroll 1
    for (uint32_t zi = warp >> 2; zi < uint32_t(kCZ); zi += kConvProducers / 128) {
        const uint32_t z = uint32_t(z0) + zi;
        const bool valid = ok && x < p.g.out_w && y < p.g.out_h && z < p.g.out_d;
        const size_t row = ((size_t(b) * p.g.out_d + z) * p.g.out_h + y) * p.g.out_w + x;
#pragma unroll 1
        for (uint32_t col0 = 0; col0 < uint32_t(BN); col0 += 16u) {
            float v[16];
            tmem_ld16(tmem + ((quarter * 32u) << 16) + zi * BN + col0, v);
            const uint32_t nb = n0 + col0;
            add_bias(p, v, nb, nb);
#pragma unroll
            for (uint32_t e = 0; e < 16u; ++e) v[e] = v[e] > 0.f ? v[e] : v[e] * slope;
            if (vec) {
                const uint32_t at = stage + lane * kPitch + col0 * 2u;
                st_shared16(at, pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                st_shared16(at + 16u, pack_bf16(v[8], v[9]), pack_bf16(v[10], v[11]), pack_bf16(v[12], v[13]),
                            pack_bf16(v[14], v[15]));
            } else if (valid) {
#pragma unroll
                for (uint32_t e = 0; e < 16u; ++e) {
                    if (nb + e >= p.n) continue;
                    if (p.mode == LBF_OUT_F32) static_cast<float*>(p.out)[row * p.ld + nb + e] = v[e];
                    else static_cast<__nv_bfloat16*>(p.out)[row * p.ld + nb + e] = __float2bfloat16_rn(v[e]);
                }
            }
        }
        if (vec) {
            __syncwarp();
            for (uint32_t k = lane; k < 32u * kParts; k += 32u) {
                const uint32_t r = k / kParts, part = k % kParts;
                const uint32_t mr = quarter * 32u + r, xr = uint32_t(x0) + (mr & 7u), yr = uint32_t(y0) + (mr >> 3);
                const uint32_t n = n0 + part * 8u;
                if (!ok || xr >= p.g.out_w || yr >= p.g.out_h || z >= p.g.out_d || n >= p.n) continue;
                const size_t vox = ((size_t(b) * p.g.out_d + z) * p.g.out_h + yr) * p.g.out_w + xr;
                *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.out) + vox * p.ld + n) =
                    ld_shared16(stage + r * kPitch + part * 16u);
            }
            __syncwarp();
        }
    }
    release(tmem, kCols);
}

// ---------------------------------------------------------------- wgrad ----

struct WgradArgs {
    Gather g;
    const uint16_t* b;
    uint32_t cb;
    uint32_t mtot;          // taps * ct
    uint32_t cps;           // K chunks per split
    uint32_t nch;           // total K chunks = ceil(rows / 64)
    float* partial;         // [split][mtot][cb]
    uint32_t* err;
};

// Mixed-radix (x, y, z, b) advance of a row index by 64.
struct Step64 {
    int ax, ay, az, ab;
};

template <int BN>
struct WgradLoader {
    const WgradArgs& p;
    SmemRing r;
    Step64 st;
    Coord rc;             // voxel of this thread's K row of the current chunk
    uint32_t base;        // first row of the current chunk
    uint32_t m_end;
    uint32_t kr, half;    // K row (t >> 1) and which 8 of its 16 pieces (t & 1)
    uint32_t tap0, ch0;   // tap and channel of the thread's first piece
    bool uniform;         // its 8 pieces are 64 contiguous channels of one tap and source
    uint32_t aoff;        // byte offset of the thread's first A piece inside a stage
    uint32_t j0;

    __device__ WgradLoader(const WgradArgs& a, const SmemRing& ring, uint32_t i0, uint32_t j0_, uint32_t c_begin,
                           uint32_t m_end_, const Step64& s64)
        : p(a), r(ring), st(s64), m_end(m_end_), j0(j0_) {
        const uint32_t t = threadIdx.x;
        kr = t >> 1;
        half = t & 1u;
        const uint32_t i = i0 + half * 64u;
        tap0 = i / p.g.ct;
        ch0 = i - tap0 * p.g.ct;
        uniform = (p.g.ct % kBK == 0) && (p.g.c1 == 0 || p.g.c0 % kBK == 0);
        aoff = half * 1024u + (kr >> 3) * 2048u + (kr & 7u) * 128u;
        base = c_begin * kBK;
        const uint32_t m = base + kr;
        rc = row_coord(p.g, m < m_end ? m : 0u);
    }

    __device__ void advance() {
        base += kBK;
        rc.x += st.ax;
        int carry = rc.x >= int(p.g.out_w);
        if (carry) rc.x -= int(p.g.out_w);
        rc.y += st.ay + carry;
        carry = rc.y >= int(p.g.out_h);
        if (carry) rc.y -= int(p.g.out_h);
        rc.z += st.az + carry;
        carry = rc.z >= int(p.g.out_d);
        if (carry) rc.z -= int(p.g.out_d);
        rc.b += st.ab + carry;
    }

    __device__ void load(uint32_t /*chunk*/, int s) {
        const uint32_t t = threadIdx.x;
        const uint32_t a = r.a(s) + aoff;
        const uint32_t sw = kr & 7u;
        const bool rowv = base + kr < m_end;
        if (uniform) {
            // Thread (kr, half) finds 128 contiguous bytes of its K row; the
            // copies are spread so that lanes 16q..16q+15 move the 16 pieces of
            // one K row (256 contiguous bytes), addresses passed by shuffles.
            const bool v = rowv && tap0 < p.g.taps;
            const uint16_t* src = p.g.src0;
            if (v) {
                int dz, dy, dx;
                tap_offsets(p.g, tap0, dz, dy, dx);
                src = chan_ptr(p.g, gather_vox(p.g, rc, dz, dy, dx), ch0);
            }
            const uint32_t lane = t & 31u, pc = lane & 15u;
            const unsigned long long sp = reinterpret_cast<unsigned long long>(src);
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t rw = 2u * i + (lane >> 4);              // K row within the warp's 16
                const int from = int(2u * rw + (pc >> 3));             // the thread holding that half
                const unsigned long long q = __shfl_sync(0xffffffffu, sp, from);
                const int vq = __shfl_sync(0xffffffffu, int(v), from);
                const uint32_t k = (t >> 5) * 16u + rw;                // K row within the chunk
                const uint32_t dst = r.a(s) + (pc >> 3) * 1024u + (k >> 3) * 2048u + (k & 7u) * 128u +
                                     (((pc & 7u) ^ (k & 7u)) << 4);
                cp_async16(dst, vq ? reinterpret_cast<const uint16_t*>(q) + 8u * (pc & 7u) : p.g.src0,
                           vq ? 16u : 0u);
            }
        } else {
            uint32_t tap = tap0, ch = ch0, cur = 0xffffffffu;
            size_t vox = 0;
#pragma unroll
            for (uint32_t jj = 0; jj < 8; ++jj) {
                const bool v = rowv && tap < p.g.taps;
                if (v && tap != cur) {
                    int dz, dy, dx;
                    tap_offsets(p.g, tap, dz, dy, dx);
                    vox = gather_vox(p.g, rc, dz, dy, dx);
                    cur = tap;
                }
                cp_async16(a + ((jj ^ sw) << 4), v ? chan_ptr(p.g, vox, ch) : p.g.src0, v ? 16u : 0u);
                ch += 8u;
                if (ch >= p.g.ct) { ch = 0; ++tap; }
            }
        }
        // B: BN/8 pieces per K row.
        constexpr uint32_t kPieces = BN / 8;
        constexpr uint32_t kRowsPerPass = kProducers / kPieces;
        constexpr uint32_t kSbo = (BN / 64) * 1024u;
        const uint32_t qn = t % kPieces;
        const uint32_t jn = j0 + qn * 8u;
#pragma unroll
        for (uint32_t it = 0; it < kBK / kRowsPerPass; ++it) {
            const uint32_t k = t / kPieces + kRowsPerPass * it;
            const uint32_t row = base + k;
            const bool v = row < m_end && jn < p.cb;
            const uint16_t* src = v ? p.b + size_t(row) * p.cb + jn : p.b;
            const uint32_t dst = r.b(s) + (qn >> 3) * 1024u + (k >> 3) * kSbo + (k & 7u) * 128u +
                                 (((qn & 7u) ^ (k & 7u)) << 4);
            cp_async16(dst, src, v ? 16u : 0u);
        }
        advance();
    }
    __device__ uint64_t adesc(int s, int kk) const { return desc_sw128(r.a(s) + 4096u * kk, 1024u, 2048u); }
    __device__ uint64_t bdesc(int s, int kk) const {
        constexpr uint32_t kSbo = (BN / 64) * 1024u;
        return desc_sw128(r.b(s) + 2u * kSbo * kk, 1024u, kSbo);
    }
};

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) wgrad_kernel(const __grid_constant__ WgradArgs p, const Step64 st) {
    extern __shared__ uint8_t smem_raw[];
    const SmemRing r = carve(smem_raw, BN * 128u);
    const uint32_t tmem = prologue(r, BN);
    const uint32_t i0 = blockIdx.x * kBM, j0 = blockIdx.y * BN;
    const uint32_t c_begin = blockIdx.z * p.cps;
    const uint32_t c_end = min(p.nch, c_begin + p.cps);
    const uint32_t m_end = min(p.g.rows, c_end * kBK);

    WgradLoader<BN> ld(p, r, i0, j0, c_begin, m_end, st);
    const uint32_t nch = c_end > c_begin ? c_end - c_begin : 0u;
    const bool ok = mainloop(ld, r, nch, tmem, idesc_bf16(kBM, BN, true, true));
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= uint32_t(kProducers / 32)) {
        release(tmem, BN);
        return;
    }
    if (!ok && nch > 0 && threadIdx.x == 0) atomicOr(p.err, LBF_ERR_MMA_TIMEOUT);

    const uint32_t i = i0 + warp * 32 + lane;
    float* out = p.partial + (size_t(blockIdx.z) * p.mtot + i) * p.cb;
#pragma unroll 1
    for (int col0 = 0; col0 < BN; col0 += 16) {
        float v[16];
        tmem_ld16(tmem + ((warp * 32u) << 16) + uint32_t(col0), v);
        if (i >= p.mtot) continue;
        for (int e = 0; e < 16; ++e) {
            const uint32_t j = j0 + col0 + e;
            if (j < p.cb) out[j] = ok ? v[e] : 0.f;
        }
    }
    release(tmem, BN);
}

__global__ void sum_partials(const float* __restrict__ part, float* __restrict__ out, size_t n, uint32_t splits) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        float s = 0.f;
        for (uint32_t k = 0; k < splits; ++k) s += part[k * n + i];
        out[i] = s;
    }
}

// -------------------------------------------------- weights, activation ----

struct PackArgs {
    const float* src;
    uint32_t dims[5];
    long long strides[5];
    uint32_t split;         // dims [0, split) make n, the others k (row-major)
    uint32_t n, k, n_pad, k_pad;
    uint16_t* dst;
};

__global__ void pack_weight_kernel(const __grid_constant__ PackArgs p) {
    const uint32_t total = p.n_pad * p.k_pad;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        uint32_t n = i / p.k_pad, k = i - n * p.k_pad;
        float v = 0.f;
        if (n < p.n && k < p.k) {
            long long at = 0;
#pragma unroll
            for (int d = 4; d >= 0; --d) {
                uint32_t& r = uint32_t(d) < p.split ? n : k;
                const uint32_t q = r / p.dims[d];
                at += (long long)(r - q * p.dims[d]) * p.strides[d];
                r = q;
            }
            v = p.src[at];
        }
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        p.dst[i] = *reinterpret_cast<const uint16_t*>(&h);
    }
}

// Backward of bias and leaky ReLU in one pass over the rows: the masked
// gradient (with y) and per-block sums of its channels.  As torch operations
// (compare, select, convert, multiply, convert, reduce) this took 216 us of a
// 64-channel 2 x 48^3 layer's backward pass, for 85 MB.  A thread keeps one
// group of 8 channels; blocks sum in FP32, the blocks' sums are added in FP64
// in block order.
constexpr int kGradThreads = 256, kGradBlocks = 148 * 4;

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__global__ void __launch_bounds__(kGradThreads)
act_grad_kernel(const uint4* __restrict__ gy, const uint4* __restrict__ y, float slope, size_t rows, uint32_t groups,
                uint4* __restrict__ out, float* __restrict__ partial) {
    extern __shared__ float acc_s[];           // [rows per block][groups * 8]
    const uint32_t per = kGradThreads / groups;
    const uint32_t r0 = threadIdx.x / groups, g = threadIdx.x - r0 * groups;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (r0 < per) {
        for (size_t r = size_t(blockIdx.x) * per + r0; r < rows; r += size_t(gridDim.x) * per) {
            const uint4 a = __ldg(&gy[r * groups + g]);
            uint32_t w[4] = {a.x, a.y, a.z, a.w};
            if (y) {
                const uint4 b = __ldg(&y[r * groups + g]);
                const uint32_t m[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float lo = bf16_lo(w[i]) * (bf16_lo(m[i]) > 0.f ? 1.f : slope);
                    const float hi = bf16_hi(w[i]) * (bf16_hi(m[i]) > 0.f ? 1.f : slope);
                    w[i] = pack_bf16(lo, hi);
                }
                out[r * groups + g] = make_uint4(w[0], w[1], w[2], w[3]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[2 * i] += bf16_lo(w[i]);
                acc[2 * i + 1] += bf16_hi(w[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) acc_s[r0 * groups * 8 + g * 8 + i] = acc[i];
    }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < groups * 8; c += kGradThreads) {
        float v = 0.f;
        for (uint32_t r = 0; r < per; ++r) v += acc_s[r * groups * 8 + c];
        partial[size_t(blockIdx.x) * groups * 8 + c] = v;
    }
}

// One warp per channel.
__global__ void __launch_bounds__(32) bias_grad_kernel(const float* __restrict__ partial, uint32_t blocks, uint32_t c,
                                                       float* __restrict__ out) {
    double v = 0.0;
    for (uint32_t b = threadIdx.x; b < blocks; b += 32) v += double(partial[size_t(b) * c + blockIdx.x]);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) out[blockIdx.x] = float(v);
}

// ----------------------------------------------------------------- host ----

int fail(const std::string& msg, int code = LBF_EINVAL) {
    lbf::set_global_error(msg);
    return code;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Validates the gather and fills the device form.  Every source voxel index
// stays inside the source grid: stride*row + tap - pad must lie in
// [-in, 2*in) on each axis so that one periodic wrap brings it back.
int make_gather(const lbf_gather& a, Gather& g, const char* who) {
    const std::string w(who);
    if (!a.src0 || (a.c1 && !a.src1)) return fail(w + ": null source");
    if (a.c0 == 0 || a.c0 % 8 || a.c1 % 8) return fail(w + ": gathered channel counts must be positive multiples of 8");
    if (!aligned16(a.src0) || (a.src1 && !aligned16(a.src1))) return fail(w + ": sources must be 16-byte aligned");
    if (a.ksize < 1 || a.ksize > 3 || a.stride < 1 || a.stride > 2) return fail(w + ": ksize must be 1..3, stride 1..2");
    if (!a.batch || !a.in_d || !a.in_h || !a.in_w || !a.out_d || !a.out_h || !a.out_w)
        return fail(w + ": empty grid");
    const uint32_t in[3] = {a.in_d, a.in_h, a.in_w}, out[3] = {a.out_d, a.out_h, a.out_w};
    for (int d = 0; d < 3; ++d) {
        const long long lo = -(long long)a.pad;
        const long long hi = (long long)a.stride * (out[d] - 1) + a.ksize - 1 - a.pad;
        if (lo < -(long long)in[d] || hi >= 2LL * in[d])
            return fail(w + ": gather reaches beyond one periodic image of the source");
    }
    const unsigned long long rows = (unsigned long long)a.batch * a.out_d * a.out_h * a.out_w;
    const unsigned long long vin = (unsigned long long)a.batch * a.in_d * a.in_h * a.in_w;
    if (rows >= (1ull << 31) || vin * (a.c0 + a.c1) >= (1ull << 40)) return fail(w + ": grid too large");
    g.src0 = static_cast<const uint16_t*>(a.src0);
    g.src1 = static_cast<const uint16_t*>(a.src1);
    g.c0 = a.c0;
    g.c1 = a.c1;
    g.ct = a.c0 + a.c1;
    g.in_d = a.in_d; g.in_h = a.in_h; g.in_w = a.in_w;
    g.out_d = a.out_d; g.out_h = a.out_h; g.out_w = a.out_w;
    g.ks = a.ksize;
    g.stride = a.stride;
    g.pad = a.pad;
    g.taps = a.ksize * a.ksize * a.ksize;
    g.rows = uint32_t(rows);
    return LBF_OK;
}

template <int BN>
int launch_igemm(const IgemmArgs& p, uint32_t n_pad, cudaStream_t s) {
    const size_t sm = smem_bytes(BN * 128u);
    cudaError_t e = cudaFuncSetAttribute(igemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm));
    if (e != cudaSuccess) return fail(std::string("lbf_igemm_run: ") + cudaGetErrorString(e), LBF_ECUDA);
    dim3 grid((p.g.rows + kBM - 1) / kBM, n_pad / BN);
    igemm_kernel<BN><<<grid, kThreads, sm, s>>>(p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(std::string("lbf_igemm_run: ") + cudaGetErrorString(e), LBF_ECUDA);
    return LBF_OK;
}

// Whether conv3_kernel takes the call: a 3x3x3 periodic convolution of at most
// kMaxConvC channels, 8 or a multiple of 16, into rows, whose tiles are not
// mostly padding.  64 channels of one source stay with igemm, which fetches a
// row's 128 bytes as one piece then: 64 -> 64 at 24^3 x 2 22 us, 27 here, at 36 x
// 48 x 48 42 and 51, at 48^3 x 2 81 and 82, at 96^3 304 and 302.  From two sources
// (32 + 32 -> 32 at 48^3 x 2 201 us, 66 here) or with fewer channels (48 -> 64 170
// and 74) it works piece by piece and loses at every size.
bool conv3_fits(const IgemmArgs& p) {
    const Gather& g = p.g;
    if (g.ks != 3 || g.stride != 1 || g.pad != 1 || g.ct > kMaxConvC || (g.ct != 8 && g.ct % 16 != 0) || g.c0 == kMaxConvC ||
        p.mode == LBF_OUT_SCATTER2_BF16 || g.in_d != g.out_d || g.in_h != g.out_h || g.in_w != g.out_w)
        return false;
    auto up = [](uint64_t n, uint64_t t) { return (n + t - 1) / t * t; };
    return up(g.out_w, kCX) * up(g.out_h, kCY) * up(g.out_d, kCZ) <= 2ull * g.out_w * g.out_h * g.out_d;
}

constexpr int kSmemMost = 227 * 1024;     // shared memory of a block, and of an SM's blocks together

// All 27 taps' weights where that leaves room for three blocks on an SM, else
// three slots of as many taps as fit into one block's shared memory.  (From 64
// outputs on tensor memory holds two blocks' accumulators, from 128 on one's: a
// further block of narrow inputs waits for its turn before it copies anything.)
constexpr TapRing conv3_ring(uint32_t groups, uint32_t bn) {
    if (groups == 1 || conv3_smem(groups, bn, TapRing{27, 1}) <= kSmemMost / 3) return TapRing{conv_taps(groups), 1};
    return conv3_smem(groups, bn, TapRing{3, 3}) <= kSmemMost ? TapRing{3, 3} : TapRing{1, 3};
}

template <int BN, int G>
int launch_conv3(const IgemmArgs& p, uint32_t n_pad, cudaStream_t s) {
    constexpr TapRing ring = conv3_ring(G, BN);
    constexpr size_t sm = conv3_smem(G, BN, ring);
    static_assert(sm <= size_t(kSmemMost), "a block's shared memory");
    static_assert(conv_taps(G) % ring.per == 0 && ring.stages <= uint32_t(kTapStages), "whole slots of taps");
    static_assert(conv3_stage_bytes(BN) <= G * kPlane + ring.per * ring.stages * G * BN * 16u,
                  "the epilogue's rows go over the tile and the weights, not over the barriers");
    cudaError_t e = cudaFuncSetAttribute(conv3_kernel<BN, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
    if (e == cudaSuccess) {
        const uint32_t tx = (p.g.out_w + kCX - 1) / kCX, ty = (p.g.out_h + kCY - 1) / kCY, tz = (p.g.out_d + kCZ - 1) / kCZ;
        const uint32_t batch = p.g.rows / (p.g.out_w * p.g.out_h * p.g.out_d);
        conv3_kernel<BN, G><<<dim3(tx * ty * tz * batch, n_pad / BN), kConvThreads, sm, s>>>(p, tx, ty, tz, ring);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return fail(std::string("lbf_igemm_run: ") + cudaGetErrorString(e), LBF_ECUDA);
    return LBF_OK;
}

template <int BN>
int launch_conv3(const IgemmArgs& p, uint32_t n_pad, cudaStream_t s) {
    if (p.g.ct == 8) return launch_conv3<BN, 1>(p, n_pad, s);
    return p.g.ct <= 16 ? launch_conv3<BN, 2>(p, n_pad, s)
                        : (p.g.ct <= 32 ? launch_conv3<BN, 4>(p, n_pad, s) : launch_conv3<BN, 8>(p, n_pad, s));
}

struct WgradPlan {
    uint32_t bn, tiles_m, tiles_n, nch, cps, splits;
    size_t bytes;
};

WgradPlan plan_wgrad(const Gather& g, uint32_t cb) {
    WgradPlan pl{};
    pl.bn = cb <= 64 ? 64 : 128;
    const uint32_t mtot = g.taps * g.ct;
    pl.tiles_m = (mtot + kBM - 1) / kBM;
    pl.tiles_n = (cb + pl.bn - 1) / pl.bn;
    pl.nch = (g.rows + kBK - 1) / kBK;
    const uint32_t tiles = pl.tiles_m * pl.tiles_n;
    // About two waves of 148 SMs, at least 8 K stages per split.
    uint32_t want = (2u * 148u + tiles - 1) / tiles;
    want = std::max(1u, std::min(want, (pl.nch + 7) / 8));
    pl.cps = (pl.nch + want - 1) / want;
    pl.splits = (pl.nch + pl.cps - 1) / pl.cps;
    pl.bytes = size_t(pl.splits) * mtot * cb * sizeof(float);
    return pl;
}

}  // namespace

extern "C" {

int lbf_igemm_run(const lbf_igemm* d, void* stream) {
    if (!d) return fail("lbf_igemm_run: null descriptor");
    IgemmArgs p{};
    int rc = make_gather(d->a, p.g, "lbf_igemm_run");
    if (rc) return rc;
    const uint32_t np = d->n_pad;
    if (!(np == 16 || np == 32 || np == 64 || (np % 128 == 0 && np > 0)))
        return fail("lbf_igemm_run: n_pad must be 16, 32, 64 or a multiple of 128");
    if (d->n == 0 || d->n > np) return fail("lbf_igemm_run: n must be in 1..n_pad");
    if (d->k_pad == 0 || d->k_pad % kBK || d->k_pad < p.g.taps * p.g.ct)
        return fail("lbf_igemm_run: k_pad must be a multiple of 64 covering ksize^3 * channels");
    if (!d->weight || !aligned16(d->weight) || !d->out || !d->err) return fail("lbf_igemm_run: null or misaligned pointer");
    if (d->out_mode > LBF_OUT_SCATTER2_BF16 || d->out_ld == 0) return fail("lbf_igemm_run: bad output mode");
    if (d->out_mode == LBF_OUT_SCATTER2_BF16 && d->n > 8u * d->out_ld)
        return fail("lbf_igemm_run: scatter output needs n <= 8 * out_ld");
    if (d->out_mode != LBF_OUT_SCATTER2_BF16 && d->n > d->out_ld) return fail("lbf_igemm_run: n exceeds out_ld");
    if (d->out_mode != LBF_OUT_F32 && !aligned16(d->out)) return fail("lbf_igemm_run: out must be 16-byte aligned");
    p.w = static_cast<const uint16_t*>(d->weight);
    p.n = d->n;
    p.k_pad = d->k_pad;
    p.bias = d->bias;
    p.out = d->out;
    p.mode = d->out_mode;
    p.ld = d->out_ld;
    p.act = d->act;
    p.slope = d->slope;
    p.err = d->err;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (conv3_fits(p)) {
        switch (np) {
            case 16: return launch_conv3<16>(p, np, s);
            case 32: return launch_conv3<32>(p, np, s);
            case 64: return launch_conv3<64>(p, np, s);
            default: return launch_conv3<128>(p, np, s);
        }
    }
    switch (np) {
        case 16: return launch_igemm<16>(p, np, s);
        case 32: return launch_igemm<32>(p, np, s);
        case 64: return launch_igemm<64>(p, np, s);
        default: return launch_igemm<128>(p, np, s);
    }
}

size_t lbf_wgrad_workspace(const lbf_wgrad* w) {
    if (!w) return 0;
    Gather g{};
    if (make_gather(w->a, g, "lbf_wgrad_workspace")) return 0;
    return plan_wgrad(g, w->cb).bytes;
}

int lbf_wgrad_run(const lbf_wgrad* w, void* stream) {
    if (!w) return fail("lbf_wgrad_run: null descriptor");
    WgradArgs p{};
    int rc = make_gather(w->a, p.g, "lbf_wgrad_run");
    if (rc) return rc;
    if (!w->b || !aligned16(w->b) || w->cb == 0 || w->cb % 8 || !w->out || !w->err)
        return fail("lbf_wgrad_run: b must be 16-byte aligned with cb a positive multiple of 8; out and err non-null");
    const WgradPlan pl = plan_wgrad(p.g, w->cb);
    if (!w->workspace || w->workspace_bytes < pl.bytes)
        return fail("lbf_wgrad_run: workspace smaller than lbf_wgrad_workspace()");
    p.b = static_cast<const uint16_t*>(w->b);
    p.cb = w->cb;
    p.mtot = p.g.taps * p.g.ct;
    p.cps = pl.cps;
    p.nch = pl.nch;
    p.partial = static_cast<float*>(w->workspace);
    p.err = w->err;
    Step64 st;
    uint32_t q = kBK;
    st.ax = int(q % p.g.out_w); q /= p.g.out_w;
    st.ay = int(q % p.g.out_h); q /= p.g.out_h;
    st.az = int(q % p.g.out_d); q /= p.g.out_d;
    st.ab = int(q);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 grid(pl.tiles_m, pl.tiles_n, pl.splits);
    cudaError_t e;
    if (pl.bn == 64) {
        const size_t sm = smem_bytes(64 * 128u);
        e = cudaFuncSetAttribute(wgrad_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm));
        if (e == cudaSuccess) wgrad_kernel<64><<<grid, kThreads, sm, s>>>(p, st);
    } else {
        const size_t sm = smem_bytes(128 * 128u);
        e = cudaFuncSetAttribute(wgrad_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm));
        if (e == cudaSuccess) wgrad_kernel<128><<<grid, kThreads, sm, s>>>(p, st);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) {
        const size_t n = size_t(p.mtot) * p.cb;
        const unsigned blocks = unsigned(std::min<size_t>((n + 255) / 256, 148u * 8u));
        sum_partials<<<blocks, 256, 0, s>>>(p.partial, w->out, n, pl.splits);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return fail(std::string("lbf_wgrad_run: ") + cudaGetErrorString(e), LBF_ECUDA);
    return LBF_OK;
}

int lbf_pack_weight(const float* src, const uint32_t dims[5], const int64_t strides[5], uint32_t split, void* dst,
                    uint32_t n_pad, uint32_t k_pad, void* stream) {
    if (!src || !dims || !strides || !dst || split < 1 || split > 4) return fail("lbf_pack_weight: invalid argument");
    PackArgs p{};
    p.src = src;
    p.split = split;
    unsigned long long n = 1, k = 1;
    for (uint32_t d = 0; d < 5; ++d) {
        if (dims[d] == 0) return fail("lbf_pack_weight: empty weight");
        p.dims[d] = dims[d];
        p.strides[d] = strides[d];
        (d < split ? n : k) *= dims[d];
    }
    if (n > n_pad || k > k_pad || (unsigned long long)n_pad * k_pad >= (1ull << 31))
        return fail("lbf_pack_weight: matrix does not fit n_pad x k_pad");
    p.n = uint32_t(n); p.k = uint32_t(k); p.n_pad = n_pad; p.k_pad = k_pad;
    p.dst = static_cast<uint16_t*>(dst);
    const unsigned blocks = std::min(148u * 4u, (n_pad * k_pad + 255u) / 256u);
    pack_weight_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(std::string("lbf_pack_weight: ") + cudaGetErrorString(e), LBF_ECUDA);
    return LBF_OK;
}

size_t lbf_act_grad_workspace(uint32_t channels) { return size_t(kGradBlocks) * channels * sizeof(float); }

int lbf_act_grad(const void* gy, const void* y, float slope, uint64_t rows, uint32_t channels, void* out, float* bias,
                 void* workspace, size_t workspace_bytes, void* stream) {
    if (!gy || !bias || !workspace || channels == 0 || channels % 8 || channels > 8u * kGradThreads || rows == 0 ||
        (y && !out) || !aligned16(gy) || (y && (!aligned16(y) || !aligned16(out))))
        return fail("lbf_act_grad: rows of 8 to 2048 channels (a multiple of 8), 16-byte aligned, and non-null results");
    if (workspace_bytes < lbf_act_grad_workspace(channels))
        return fail("lbf_act_grad: workspace smaller than lbf_act_grad_workspace()");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint32_t groups = channels / 8, per = kGradThreads / groups;
    const unsigned blocks = unsigned(std::min<uint64_t>(kGradBlocks, (rows + per - 1) / per));
    act_grad_kernel<<<blocks, kGradThreads, size_t(per) * channels * sizeof(float), s>>>(
        static_cast<const uint4*>(gy), static_cast<const uint4*>(y), slope, rows, groups, static_cast<uint4*>(out),
        static_cast<float*>(workspace));
    bias_grad_kernel<<<channels, 32, 0, s>>>(static_cast<const float*>(workspace), blocks, channels, bias);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(std::string("lbf_act_grad: ") + cudaGetErrorString(e), LBF_ECUDA);
    return LBF_OK;
}

void lbf_operator_info(uint32_t out[4]) {
    out[0] = kBM;
    out[1] = kBK;
    out[2] = kStages;
    out[3] = kThreads;
}

}  // extern "C"
