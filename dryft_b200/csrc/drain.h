// Which copies of a ring may still be in flight, and waiting for them: plain C++ for host and device, so that it can be tested on
// the CPU.
//
// Copy i of a ring goes into stage i % stages and completes phase i / stages of that stage's barrier.  A stage is filled
// again only once its copy was used, so no more than the last `stages` copies are on their way.  `landed(stage, parity)` is the
// barrier's test of a phase: it tells a phase that has ended from the one after it by the phase's parity, so the parity to
// ask for is the one of the copy -- a stage that is asked for either parity always answers yes.
#pragma once

#ifdef __CUDACC__
#define DRYFT_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define DRYFT_HOST_DEVICE inline
#endif

// Waits until every copy that was issued has landed; false when `expired()` says so first.
template <typename Landed, typename Expired>
DRYFT_HOST_DEVICE bool ring_drain(int issued, int stages, Landed landed, Expired expired) {
  for (int i = issued > stages ? issued - stages : 0; i < issued; ++i)
    while (!landed(i % stages, (unsigned)((i / stages) & 1)))
      if (expired()) return false;
  return true;
}
