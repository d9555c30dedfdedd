// amrlbm_wait.h - what a CTA does when a bulk copy does not land in time, apart
// from the instructions that wait, so that a host compiler takes it too
// (tests/test_copy_waits.py).
#pragma once

#ifdef __CUDACC__
#define AMR_WAIT_FN __device__ __forceinline__
#else
#define AMR_WAIT_FN inline
#endif

// The copies behind a CTA's two mbarriers. A barrier's parity advances only once
// its completion has been seen: a wait on the other parity asks for the phase
// before and returns at once, whether the copy has landed or not.
struct CopyWaits {
    unsigned parity = 0;  // bit b: parity of barrier b's next completion

    // Bounded wait for barrier b. wait_on(b, parity): whether barrier b completed
    // in time; any(x): x of some thread of the CTA. Every thread gets the same
    // answer. On false every thread has waited (bounded) once more for all the
    // barriers of mask `in_flight`, so that no copy writes into shared memory
    // that the CTA has given up, and the caller leaves without using what did
    // not land.
    template <class WAIT, class ANY>
    AMR_WAIT_FN bool landed(int b, unsigned in_flight, WAIT wait_on, ANY any) {
        if (any(!wait_on(b, (parity >> b) & 1u))) {
            for (int i = 0; in_flight >> i; ++i)
                if ((in_flight >> i) & 1u) wait_on(i, (parity >> i) & 1u);
            return false;
        }
        parity ^= 1u << b;
        return true;
    }
};
