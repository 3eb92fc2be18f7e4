/* The tile kernel for launches whose tiles are all of one shape (a handle's
 * call, an array's, the fused front end): registers for that shape alone (4 to
 * 152 bytes of spills). Compiled once
 * per nchan, 2^ONE_LOGM, by the Makefile (an object each, built side by side);
 * without ONE_LOGM it is the table of them.
 *
 * One stream of 8,388,301 samples, nchan 1024, 2x, 16 taps: 204.5 us through the
 * kernel of every shape, 196.4 here; eight elements at nchan 2048: 141, 134. */
#ifdef ONE_LOGM
#include "pfb_kernel.cuh"

#define PASTE2(a, b) a##b
#define PASTE(a, b) PASTE2(a, b)

namespace {

template <int KEY>
struct OneShape {
    static __device__ __forceinline__ void carry(const Src &src, float2 *dst, long long from, long long len) {
        carry_copy<NT>(src, dst, from, len);
    }
    static __device__ __forceinline__ void run(int key, const atkb_job &J, const atkb_bank &SB, long long h0,
                                               int nvalid, double2 *sm, float2 *to) {
        if (key == KEY) run_tile<KEY>(J, SB, h0, nvalid, sm, to);
    }
};

template <int KEY>
__global__ void __launch_bounds__(NT, 2)
pfb_tiles_one(const atkb_job *__restrict__ jobs, const int *__restrict__ tile_start,
              const atkb_carry *__restrict__ carries, int njobs, const int *__restrict__ d_njobs, int *counters) {
    tiles_loop<OneShape<KEY>>(jobs, tile_start, carries, njobs, d_njobs, counters);
}

}  // namespace

extern "C" const void *PASTE(atkb_pfb_one_, ONE_LOGM)(int shape) {
    switch (shape) {
#define S(n) case n: return (const void *)pfb_tiles_one<16 * n + ONE_LOGM>;
    S(0) S(1) S(2) S(3)
#if ONE_LOGM <= 10
    S(5) S(6)
#endif
#undef S
    default: return nullptr;
    }
}

extern "C" unsigned PASTE(atkb_pfb_one_fault_, ONE_LOGM)(void) {
#ifdef ATKB_DEBUG_BOUNDS
    return take_debug_fault();
#else
    return 0;
#endif
}

#else
#include "internal.h"

#define EACH(X) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)
#define DECLARE(L)                                          \
    extern "C" const void *atkb_pfb_one_##L(int shape);     \
    extern "C" unsigned atkb_pfb_one_fault_##L(void);
EACH(DECLARE)

extern "C" const void *atkb_pfb_one(int key) {
    switch (key & 15) {
#define GET(L) case L: return atkb_pfb_one_##L(key >> 4);
        EACH(GET)
    default: return nullptr;
    }
}

extern "C" unsigned atkb_pfb_one_fault(void) {
#define OR(L) | atkb_pfb_one_fault_##L()
    return 0u EACH(OR);
}
#endif
