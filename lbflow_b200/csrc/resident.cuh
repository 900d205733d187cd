// Many time steps of one small geometry in one launch.
//
// A geometry whose nodes all fit on the GPU at once (one thread per fluid
// node) is stepped by a single cooperative launch: every thread keeps its
// node's pull sources in registers for all steps, and a post-collision
// population travels to its one reader as a word that holds the value and the
// number of the step that wrote it, written and read as one access.  The
// reader polls the word itself until the step it needs appears, so there is
// no launch, barrier, fence or flag between steps: a step costs one store to
// L2, one load from L2 and the collision.
//
// Two word arrays alternate.  Overwriting is safe without further
// synchronisation: the word that node x writes at step s is read by x + e at
// step s + 1; x writes that array again at step s + 2, after it has read, at
// step s + 2, what x + e computed at step s + 1 from all its inputs, that word
// among them (links are symmetric; a bounced population is read by its own
// node).
//
// Bound by the L2 round trip (store to the reader's poll) and the collision's
// dependent chain.  Microseconds per step, one launch per step (with
// programmatic dependent launch) -> here: D2Q9 FP64 48x40 (1 k nodes) 3.6 ->
// 1.3, 300x300 (45 k) 3.5 -> 1.9; D3Q19 FP64 48^3 (24 k) 4.7 -> 2.6, 64x64x80
// (72 k) 6.6 -> 4.4; FP32 64^3 (58 k) 3.8-5.3 -> 2.5, 80x80x90 (127 k) 6.0 ->
// 4.4; FP16 80x80x78 (110 k) 6.5 -> 4.1.  At the largest geometry that fits it
// is still the faster form, so it is used whenever the geometry fits.
//
// Between launches the populations are in the engine's ordinary array: the
// first step reads it, the last step writes the other one.  Every wait is
// bounded; on timeout the kernel sets kErrWait and returns, the state is then
// undefined, and later launches return at their first wait until the state is
// initialised anew.
#pragma once
#include "kernels.cuh"

namespace lbf {

constexpr long long kResidentWait = 4000000000LL;   // default limit of a wait: clock cycles, about 2 s

struct Resident {
    void* words;        // [2][Q - 1][nfp] tagged words
    uint32_t tag0;      // step number before the launch's first step
    uint32_t steps;     // >= 2
    long long wait;     // limit of a wait, in clock cycles
};

// A population and the number of the step that wrote it, moved as one access.
struct Word128 { unsigned long long value, tag; };

__device__ __forceinline__ void put_word(Word128* p, double v, uint32_t tag)
{
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}\n"
                 ::"l"(p), "l"(__double_as_longlong(v)), "l"((unsigned long long)tag) : "memory");
}
__device__ __forceinline__ uint32_t get_word(const Word128* p, double& v)
{
    long long lo, hi;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}\n"
                 : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    v = __longlong_as_double(lo);
    return (uint32_t)hi;
}
__device__ __forceinline__ void put_word(unsigned long long* p, uint32_t bits, uint32_t tag)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)tag << 32) | bits) : "memory");
}
__device__ __forceinline__ uint32_t get_word(const unsigned long long* p, uint32_t& bits)
{
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    bits = (uint32_t)w;
    return (uint32_t)(w >> 32);
}

// Payload of a word by storage type.
template <class S> struct Payload;
__device__ __forceinline__ uint32_t peek_word(const void* p)
{
    uint32_t t;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(t) : "l"(p) : "memory");
    return t;
}
template <> struct Payload<StoreF64> {
    using W = Word128;
    __device__ static uint32_t peek(const W* p) { return peek_word(&p->tag); }
    __device__ static uint32_t get(const W* p, int, double& v) { return get_word(p, v); }
    __device__ static void put(W* p, double v, int, uint32_t tag) { put_word(p, v, tag); }
};
template <class L> struct Payload<StoreF32<L>> {
    using W = unsigned long long;
    __device__ static uint32_t peek(const W* p) { return peek_word(reinterpret_cast<const uint32_t*>(p) + 1); }
    __device__ static uint32_t get(const W* p, int, float& v)
    {
        uint32_t b;
        const uint32_t t = get_word(p, b);
        v = __uint_as_float(b);
        return t;
    }
    __device__ static void put(W* p, float v, int, uint32_t tag) { put_word(p, __float_as_uint(v), tag); }
};
template <class L, class H> struct Payload<StoreShifted16<L, H>> {
    using W = unsigned long long;
    __device__ static uint32_t peek(const W* p) { return peek_word(reinterpret_cast<const uint32_t*>(p) + 1); }
    __device__ static uint32_t get(const W* p, int q, float& v)
    {
        uint32_t b;
        const uint32_t t = get_word(p, b);
        v = StoreShifted16<L, H>::from_bits((uint16_t)b, q);
        return t;
    }
    __device__ static void put_bits(W* p, uint32_t bits, uint32_t tag) { put_word(p, bits, tag); }
};

// One warp per block spreads a geometry evenly over the SMs (48^3 FP64, 24 k
// nodes: 2.62 us per step, 2.89 with 128-thread blocks).  Blocks per SM the
// kernel is compiled for set the largest geometry it takes (times 148 x 32
// nodes): FP64 D3Q19 16 (128 registers; at 20 it spills and 48^3 slows from
// 2.9 to 3.3 us), FP32 arithmetic 28, D2Q9 20 and 32.
constexpr unsigned kResidentThreads = 32;
template <class L, class S> struct ResidentBlocks {
    static constexpr bool f64 = sizeof(typename S::R) == 8;
    static constexpr int value = L::D == 2 ? (f64 ? 20 : 32) : (f64 ? 16 : 28);
};

// Whole warp, while waiting: true once the wait has lasted `limit` or another
// block gave up.
__device__ __forceinline__ bool resident_late(long long& t0, long long limit, uint32_t* err)
{
    const long long t = clock64();
    if (t0 == 0) t0 = t;
    const bool late = t - t0 >= limit || (*(volatile uint32_t*)err & kErrWait);
    if (!__any_sync(0xffffffffu, late)) return false;
    atomicOr(err, kErrWait);
    return true;
}

// All steps of a call: out (macroscopic fields wanted) applies to the last.
// P.seed: for 16-bit storage the number of the first step, from which each
// step's rounding seed follows as in the one-step launches.
template <class L, class S>
__global__ void __launch_bounds__(kResidentThreads, ResidentBlocks<L, S>::value)
scsp_resident(const Grid g, const Force F, const ScspParams P0, const typename S::T* fin,
              typename S::T* __restrict__ fout, const Resident r, Macros mo, const int out,
              uint32_t* __restrict__ err)
{
    using R = typename S::R;
    using PL = Payload<S>;
    using W = typename PL::W;
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x;
    // Lanes past the last node follow it, without storing.
    const bool live = i0 < g.nf;
    const uint32_t i = live ? i0 : g.nf - 1;
    const uint32_t nfp = g.nfp;
    int x, y, z;
    unpack(__ldg(&g.coord[i]), x, y, z);
    uint32_t off[L::Q];
    {
        const uint32_t mask = pull_sources<L, (sizeof(R) == 4)>(g, x, y, z, off);
#pragma unroll
        for (int q = 1; q < L::Q; ++q) {
            const bool fluid = (mask >> q) & 1u;
            off[q] = (uint32_t)((fluid ? q : L::op(q)) - 1) * nfp + (fluid ? off[q] : i);
        }
    }
    R f[L::Q];
    f[0] = S::load(fin + i, 0, R(P0.rho0));
#pragma unroll
    for (int q = 1; q < L::Q; ++q) f[q] = S::load(fin + (nfp + off[q]), q, R(P0.rho0));
    ScspParams P = P0;
    const size_t half = (size_t)(L::Q - 1) * nfp;
    for (uint32_t s = 0;; ++s) {
        const bool last = s + 1 == r.steps;
        if (S::dither) P.seed = ((P0.seed + s) * 2654435761u) | 1u;
        scsp_collide<L, S>(g, F, P, i, f, mo, last ? out : 0, err);
        if (last) break;
        const uint32_t tag = r.tag0 + s + 1;
        W* const dst = static_cast<W*>(r.words) + (tag & 1u ? half : 0);
        if constexpr (S::dither) {
            uint16_t b[L::Q];
            S::round(f, b, P, i);
            f[0] = S::from_bits(b[0], 0);
#pragma unroll
            for (int q = 1; q < L::Q; ++q) if (live) PL::put_bits(dst + ((uint32_t)(q - 1) * nfp + i), b[q], tag);
        } else {
#pragma unroll
            for (int q = 1; q < L::Q; ++q) if (live) PL::put(dst + ((uint32_t)(q - 1) * nfp + i), f[q], q, tag);
        }
        // D3Q19: the warp polls one word per lane, first an arbitrary one,
        // then one that a pass over all of them found missing: polling all 18
        // loads L2 enough to delay the words that are waited for (56^3 FP64:
        // 3.5 us per step, 3.2 so).  D2Q9 with its 8 words is faster polling
        // them all (48x40: 1.17 against 1.27).  The lanes stay together
        // (votes): alone, each would make passes of its own (16^3: 6.9 us).
        uint32_t miss = L::D == 2 ? 0xffffffffu : off[L::Q - 1];
        long long t0 = 0;
        for (;;) {
            if constexpr (L::D == 3) {
                uint32_t n = 0;
                while (__any_sync(0xffffffffu, miss != 0xffffffffu && PL::peek(dst + miss) != tag))
                    if ((++n & 255u) == 0 && resident_late(t0, r.wait, err)) return;
            }
            miss = 0xffffffffu;
#pragma unroll
            for (int q = 1; q < L::Q; ++q)
                if (PL::get(dst + off[q], q, f[q]) != tag) miss = off[q];
            if (!__any_sync(0xffffffffu, miss != 0xffffffffu)) break;
            if (resident_late(t0, r.wait, err)) return;
        }
    }
    if (live) scsp_store<L, S>(g, P, fout, i, f, nullptr);
}

}  // namespace lbf
