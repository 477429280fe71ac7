// Which copies of a ring of shared-memory stages may still be under way when a block gives up, for kernels that count every
// copy with an mbarrier a stage: piece c lies in stage c % stages, and its arrival completes the barrier's phase c / stages. A
// wait names the parity of the phase it is for; with the wrong one it returns at once on the phase before, and the block would
// end with a copy still to land in shared memory that another block may own by then.
#pragma once

#ifdef __CUDACC__
#define CELEG_RING_INLINE __device__ __forceinline__
#else
#define CELEG_RING_INLINE inline
#endif

namespace celeg_b200 {

// wait(stage, parity) for the pieces from `first` up to `brought` (not included): every piece before `first` has been waited
// for. No stage without a copy under way is waited for.
template <typename Wait>
CELEG_RING_INLINE void drain_ring(int first, int brought, int stages, Wait wait) {
    for (int c = first; c < brought; ++c) wait(c % stages, (unsigned)(c / stages) & 1u);
}

}  // namespace celeg_b200
