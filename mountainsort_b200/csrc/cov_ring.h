// When a converter group of the tensor-core covariance may take stage g of its ring: the
// MMAs have read the planes of stage g - stages from the slot, and the slot's tiles have
// landed.
//
// The order of the two waits matters.  A group takes every other stage, and the ring's
// stages are odd in number, so the slot's last stage was the other group's: this group has
// not waited for its tiles.  Where they have not landed either, the tiles' barrier is one
// phase further back than the parity test supposes, and the test takes the phase before
// that for the one it asks for.  (The groups took stages whose tiles were still on their
// way, about one call in ten when several recordings shared the GPU: wrong covariances, and
// copies that landed after their CTA had left.)  The planes' barrier cannot be behind: the
// group waited for stage g - 2 - stages there, and the MMAs complete in order.  Once it
// shows stage g - stages done, that stage's tiles had landed, and the tiles' barrier is in
// the phase of stage g or past it.
#ifndef MS3_COV_RING_H
#define MS3_COV_RING_H

#include <cstdint>

#ifdef __CUDACC__
#define MS3_RING_D __device__ __forceinline__
#else
#define MS3_RING_D inline
#endif

namespace ms3gpu {

// phase: of stage g in its slot, (g / stages) & 1.  The waits take a parity and return
// whether that phase is over.
template <class PlanesRead, class TilesLanded>
MS3_RING_D bool converter_may_take(int64_t g, int stages, uint32_t phase, PlanesRead planes_read,
                                   TilesLanded tiles_landed) {
    return (g < stages || planes_read(phase ^ 1u)) && tiles_landed(phase);
}

}  // namespace ms3gpu

#endif
