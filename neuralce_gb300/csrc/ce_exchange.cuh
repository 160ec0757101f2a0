// Slot exchange of one ladder, by one warp: the rule that the chunk kernels run at their end and ce_exchange_kernel in a
// launch of its own.  The memory of other lanes is read only past a __syncwarp(): shuffles and warp reductions order no
// memory.  (Plain C++ but for the warp primitives, so that a host program that supplies those can run it lane by lane.)
#pragma once
#include <math.h>

#include "common.cuh"

namespace nce {

struct ExArgs {
    int32_t R; const double *E; double E_scale;
    const float *beta_slot; int32_t *rep_of_slot, *slot_of_rep; const int32_t *ladder_id; int64_t *n_ex;
    uint64_t seed; int64_t g_end; const double *ex_u;   // host uniforms (rounds, R / 2) or null: Philox
    int32_t parity, rounds;                             // host parities, a bit a round (with ex_u)
    double *E_samples; int64_t row;                     // the last sample row is rewritten in the new order (null: none)
};

// The pairs of a round are disjoint, so a lane takes a pair: one thread walking them spent about 1 us a pair on dependent
// loads and a float64 logarithm (256 replicas of 131,072 sites, chunks of 300 steps: 1,462 -> 1,196 us; 16 of 256 sites, 10
// steps: 77 -> 63 us, on the step-by-step kernel).
__device__ __forceinline__ void exchange_warp(const ExArgs &x, int lane) {
    const int R = x.R;
    const uint32_t k0 = (uint32_t)x.seed, k1 = (uint32_t)(x.seed >> 32);
    const uint32_t c0 = (uint32_t)x.g_end, c1 = (uint32_t)((uint64_t)x.g_end >> 32);
    const int npair = R / 2;                            // ceil((R-1)/2)
    int nswap = 0;
    for (int q = 0; q < x.rounds; ++q) {
        const uint32_t cq = 0xFFFFFFFFu - 2u * (uint32_t)q;
        const int parity = x.ex_u ? ((x.parity >> q) & 1) : (int)(philox4x32(c0, c1, cq, 0u, k0, k1).x & 1u);
        for (int k = lane; 2 * k < R - 1; k += 32) {
            const int a = 2 * k + parity, b = a + 1;
            if (b >= R || x.ladder_id[a] != x.ladder_id[b]) continue;
            const int32_t ra = __ldcg(x.rep_of_slot + a), rb = __ldcg(x.rep_of_slot + b);
            const double Ea = __ldcg(x.E + ra) * x.E_scale, Eb = __ldcg(x.E + rb) * x.E_scale;
            const double log_acc = ((double)x.beta_slot[b] - (double)x.beta_slot[a]) * (Eb - Ea);
            double u;
            if (x.ex_u) u = x.ex_u[(size_t)q * npair + k];
            else { const u32x4 w = philox4x32(c0, c1, cq - 1u, (uint32_t)k, k0, k1); u = draw_u01(w.x, w.y); }
            if (log(u) < log_acc) { x.rep_of_slot[a] = rb; x.rep_of_slot[b] = ra; ++nswap; }
        }
        __syncwarp();                                   // the next round, and the slots below, read what other lanes swapped
    }
    nswap = __reduce_add_sync(0xffffffffu, nswap);
    if (lane == 0) *x.n_ex += nswap;
    for (int q = lane; q < R; q += 32) {
        const int32_t rq = __ldcg(x.rep_of_slot + q);
        x.slot_of_rep[rq] = q;
        if (x.E_samples) x.E_samples[x.row * R + q] = __ldcg(x.E + rq);
    }
}

// Chunk end, called by one whole warp of each replica (the cluster's first CTA) once its outputs are written: the last
// replica of the job to arrive performs the job's slot exchange, advances the device step counter and re-arms the counter.
// No thread waits for another, so the chunk kernel never depends on its CTAs running at the same time.
template <typename Job>
__device__ void fused_chunk_end(const Job &jb, int64_t g0, int lane) {
    int last = 0;
    if (lane == 0) {
        __threadfence();                                // this replica's energy is visible before it is counted
        last = atomicAdd(jb.ex_sync, 1) == jb.R - 1;
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();                                    // lane 0 has seen every replica's count;
    __syncwarp();                                       // so every lane sees what they wrote before it
    const int64_t g_end = g0 + jb.n_steps;
    if (lane == 0 && jb.step_dev) *const_cast<int64_t *>(jb.step_dev) = g_end;   // every CTA of the job has read it by now
    if ((jb.ex_flags & 1) && jb.R > 1) {
        ExArgs x;
        x.R = jb.R; x.E = jb.E; x.E_scale = 1.0; x.beta_slot = jb.beta_slot; x.rep_of_slot = jb.rep_of_slot;
        x.slot_of_rep = jb.slot_of_rep; x.ladder_id = jb.ladder_id; x.n_ex = jb.n_ex; x.seed = jb.seed; x.g_end = g_end;
        x.ex_u = jb.ex_u; x.parity = (jb.ex_flags >> 1) & 1; x.rounds = 1;
        const bool rewrite = jb.E_samples && jb.n_steps > 0 && jb.n_steps % jb.sample_interval == 0;
        x.E_samples = rewrite ? jb.E_samples : nullptr;
        x.row = rewrite ? jb.n_steps / jb.sample_interval - 1 : 0;
        exchange_warp(x, lane);
    }
    if (lane == 0) *jb.ex_sync = 0;
}

}  // namespace nce
