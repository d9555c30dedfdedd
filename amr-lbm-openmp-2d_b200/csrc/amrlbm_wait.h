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

    // Bounded waits for the barriers of mask `wait`. wait_on(b, parity): whether
    // barrier b completed in time; any(x): x of some thread of the CTA. Every
    // thread gets the same answer. On false every thread has waited (bounded)
    // once more for all the barriers of mask `in_flight`, so that no copy writes
    // into shared memory that the CTA has given up, and the caller leaves
    // without using what did not land.
    template <class WAIT, class ANY>
    AMR_WAIT_FN bool landed(unsigned wait, unsigned in_flight, WAIT wait_on, ANY any) {
        bool late = false;
        for (int b = 0; b < 2; ++b)
            if ((wait >> b) & 1u) late |= !wait_on(b, (parity >> b) & 1u);
        if (any(late)) {
            for (int b = 0; b < 2; ++b)
                if ((in_flight >> b) & 1u) wait_on(b, (parity >> b) & 1u);
            return false;
        }
        parity ^= wait;
        return true;
    }
};
