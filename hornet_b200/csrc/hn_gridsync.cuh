// Grid barrier of cooperative launches (all CTAs resident), with a bounded
// wait.
#pragma once

#include "hn_internal.cuh"

namespace hn {

// In device memory, zeroed once; a launch that ends without a timeout leaves
// it ready for the next.  After a timeout `arrive` may count CTAs that have
// left, and a barrier counted on from it would open with CTAs still outside.
// So the wait that gives up sets kGridDead in it, which no barrier clears:
// every later barrier of this launch, and of launches queued behind it, is
// refused until the host zeroes the struct.
struct GridBar {
    unsigned arrive;   // CTAs at the barrier, kGridDead
    unsigned gen;      // barriers passed
    unsigned beat;     // moved by CTAs that work on while others wait (grid_progress)
    unsigned pad;
};
constexpr unsigned kGridDead = 1u << 31;

// Work of one CTA or warp between two barriers that may take longer than a
// wait's limit tells the others, every few milliseconds, that it goes on.
__device__ __forceinline__ void grid_progress(GridBar* bar) { atomicAdd(&bar->beat, 1u); }

// One thread of each CTA, between two __syncthreads.  The last CTA to arrive
// runs `seal` before it opens the barrier.  `gen` is the CTA's count of
// barriers passed, first read from bar->gen before the CTA's first arrival.
// `limit`: polls without progress (neither the barrier nor `beat` moved) before
// a wait gives up (the grid.wait_polls knob; its default is seconds).
// Writes before the barrier are visible to every CTA after it.  False: a wait
// gave up, here or in another CTA, and the CTA must leave the kernel.
template <typename Seal>
__device__ __forceinline__ bool grid_barrier(GridBar* bar, unsigned& gen, unsigned limit,
                                             Seal seal) {
    bool ok = true;
    __threadfence();
    const unsigned before = atomicAdd(&bar->arrive, 1u);
    if (before == gridDim.x - 1) {
        __threadfence();
        seal();
        atomicSub(&bar->arrive, gridDim.x);   // (not a store: kGridDead stays)
        __threadfence();
        atomicAdd(&bar->gen, 1u);
    } else if (before & kGridDead) {
        ok = false;
    } else {
        unsigned polls = 0, beat = 0;
        while (*(volatile unsigned*)&bar->gen == gen) {
            if (++polls >= 64) __nanosleep(40);
            if ((polls & 1023u) == 0) {
                const unsigned b = *(volatile unsigned*)&bar->beat;
                if (b != beat) {
                    beat = b;
                    polls = 64;
                }
                if (polls >= limit || (*(volatile unsigned*)&bar->arrive & kGridDead)) {
                    atomicOr(&bar->arrive, kGridDead);
                    ok = false;
                    break;
                }
            }
        }
    }
    __threadfence();
    gen++;
    return ok;
}

}  // namespace hn
