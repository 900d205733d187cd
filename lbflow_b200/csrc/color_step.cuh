// Launches of one two-phase step for one storage type.  Each storage type is a
// translation unit of its own (color_fp64.cu, ...): together they take ptxas
// ten minutes.
#pragma once
#include "internal.h"
#include "../../include/lbflow.h"

namespace lbf {

namespace {
template <class L, class S, int COLL, bool FILM>
void run_step(bool pull, int out, const ColorLaunch& a)
{
    using T = typename S::T;
    const T* fin = static_cast<const T*>(a.fin);
    T* fout = static_cast<T*>(a.fout);
    const unsigned threads = 128, blocks = blocks_for(a.g.nf, threads);
    if (blocks == 0) return;
    const unsigned zb = blocks_for(a.zh.n, threads);
    const double rb = a.P.rho_ref[0];
    if (pull)
        launch_pdl(color_phase<L, S, true, FILM>, blocks, threads, a.stream, a.g, a.film, fin, a.dens, a.phid, a.err, rb);
    else
        color_phase<L, S, false, false><<<blocks, threads, 0, a.stream>>>(a.g, a.film, fin, a.dens, a.phid, a.err, rb);
    // Zou-He boundary nodes (PB/VB): their phase from the rebuilt populations
    // before pass 2 reads it, and their collision after pass 2 (overwriting).
    if (pull && zb)
        launch_pdl(color_zou_he_phase<L, S, FILM>, zb, threads, a.stream, a.g, a.film, a.zh, fin, a.phid, a.err, rb);
    if (!pull && zb && (out & kOutAdjacent))
        color_zou_he_record<L, S><<<zb, threads, 0, a.stream>>>(a.g, a.zh, fin, rb);
    if (pull)
        launch_pdl(color_collide<L, S, COLL, true, FILM>, blocks, threads, a.stream, a.g, a.film, a.F, a.P, a.W, fin,
                   fout, a.dens, a.phid, a.mo, out, a.err);
    else
        color_collide<L, S, COLL, false, false><<<blocks, threads, 0, a.stream>>>(
            a.g, a.film, a.F, a.P, a.W, fin, fout, a.dens, a.phid, a.mo, out, a.err);
    if (pull && zb)
        launch_pdl(color_zou_he_collide<L, S, COLL, FILM>, zb, threads, a.stream, a.g, a.film, a.F, a.P, a.W, a.zh, fin,
                   fout, a.phid, a.mo, out, a.err);
}

template <class L, class S, int COLL>
void dispatch(bool pull, int out, const ColorLaunch& a)
{
    // Half films: the film-aware gathers only where the geometry has films
    // (FP64 and FP32 storage; the engine refuses films with 16-bit storage).
    if constexpr (IsPacked<S>::value) run_step<L, S, COLL, false>(pull, out, a);
    else if (a.film.bits[0]) run_step<L, S, COLL, true>(pull, out, a);
    else run_step<L, S, COLL, false>(pull, out, a);
}

template <class L, class S>
void dispatch_coll(int collision, bool pull, int out, const ColorLaunch& a)
{
    if (collision == LBF_MRT) dispatch<L, S, 1>(pull, out, a);
    else dispatch<L, S, 0>(pull, out, a);
}
}  // namespace

}  // namespace lbf
