// Grid barrier of cooperative launches (all CTAs resident), with a bounded
// wait.
#pragma once

#include "hn_internal.cuh"

namespace hn {

// In device memory, zeroed once; a launch that ends without a timeout leaves
// it ready for the next.
struct GridBar {
    unsigned arrive;   // CTAs at the barrier
    unsigned gen;      // barriers passed
    unsigned beat;     // moved by a CTA that works on while the others wait
    unsigned pad;
};

// Polls without progress (neither the barrier nor `beat` moved) before a wait
// gives up: seconds.
constexpr unsigned kGridWait = 1u << 24;

// One thread of each CTA, between two __syncthreads.  The last CTA to arrive
// runs `seal` before it opens the barrier.  `gen` is the CTA's count of
// barriers passed, first read from bar->gen before the CTA's first arrival.
// Writes before the barrier are visible to every CTA after it.  False: the
// wait gave up, and the CTA must leave the kernel.
template <typename Seal>
__device__ __forceinline__ bool grid_barrier(GridBar* bar, unsigned& gen, Seal seal) {
    bool ok = true;
    __threadfence();
    if (atomicAdd(&bar->arrive, 1u) == gridDim.x - 1) {
        __threadfence();
        seal();
        bar->arrive = 0;
        __threadfence();
        atomicAdd(&bar->gen, 1u);
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
                if (polls >= kGridWait) {
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
