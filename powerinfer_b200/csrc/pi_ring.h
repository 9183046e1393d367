// Rings of shared-memory stages: which phase of a stage's barrier its last copies belong to.  Plain C++, so that a program without CUDA can
// walk it.
#pragma once

#ifdef __CUDACC__
#define PI_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PI_HOST_DEVICE inline
#endif

namespace pi {

// Stages 0 .. issued - 1 went to the slots in turn, and each use of a slot is one phase of its barrier: the parity of the phase that the last
// use of `slot` completes, -1 where it had none.  (A barrier says that the phase BEFORE the current one is over for the other parity,
// from the start on: a wait for "either parity" waits for nothing.)
PI_HOST_DEVICE int ring_last_parity(int issued, int slots, int slot) { return slot < issued ? (issued - 1 - slot) / slots & 1 : -1; }

}  // namespace pi
