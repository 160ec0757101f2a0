// Step bookkeeping of the windowed kernel (ce_window.cuh): which proposals are drawn ahead of a window and which steps of it
// are sampled.  Steps are 32-bit and a chunk may have 2^31 - 2 of them: a signed sum past the chunk's end would turn negative
// and draw or sample steps that do not exist.  Plain C++, so that the host can run it.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define NCE_STEP_FN __host__ __device__ __forceinline__
#else
#define NCE_STEP_FN inline
#endif

namespace nce {

constexpr int kWinRing = 128;            // proposals in flight (a window reaches 32 steps ahead, drawn 64 ahead)

// ring slot of step s + i
NCE_STEP_FN int win_slot(int32_t s, int i) { return (int)(((uint32_t)s + (uint32_t)i) & (uint32_t)(kWinRing - 1)); }

// Steps drawn so far are counted without a sign and past the chunk's end too: at most 2^31 + 126.  Whether the window that
// starts at step s draws the next 32 (fewer than 96 steps are drawn ahead of its start, so at most kWinRing are in the ring
// afterwards), and whether step drawn + lane is one of the chunk's T.
NCE_STEP_FN bool win_draws(uint32_t drawn, int32_t s) { return drawn - (uint32_t)s < 96u; }
NCE_STEP_FN bool win_in_chunk(uint32_t drawn, int lane, int32_t T) { return drawn + (uint32_t)lane < (uint32_t)T; }

// Sampling every si steps: `left` is the number of steps from the window's start up to and including the next sampled one (1 ..
// si).  Whether step i (from 0) of a window that has decided `limit` steps is sampled, and `left` at the start of the next.
NCE_STEP_FN bool win_samples(int32_t left, int32_t si, int i, int limit) {
    return i < limit && i + 1 >= left && (i + 1 - left) % si == 0;
}
NCE_STEP_FN int32_t win_left(int32_t left, int32_t si, int limit) {
    left -= limit;
    return left > 0 ? left : left + ((-left) / si * si + si);
}

}  // namespace nce
