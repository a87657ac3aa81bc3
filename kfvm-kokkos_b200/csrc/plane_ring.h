// plane_ring.h -- the state planes of a block that marches along z over the cells of planes
// k0 .. k1 - 1, which read two planes on either side: planes k0 - 2 .. last (= k1 + 1) pass
// through a ring of slots.  Usable from device code (recon_sym.cu: TMA loads, one mbarrier per
// slot, one thread issues and every thread waits) and from the host.
#pragma once

#ifdef __CUDACC__
#define KFVM_RING_HD __host__ __device__ __forceinline__ constexpr
#else
#define KFVM_RING_HD constexpr
#endif

namespace kfvm {

template <int RING>
struct PlaneRing {
  // slot of plane p, and the phase of the slot's barrier that its load completes
  KFVM_RING_HD static int slot(int k0, int p) { return (p - k0 + 2) % RING; }
  KFVM_RING_HD static unsigned parity(int k0, int p) { return (unsigned)((p - k0 + 2) / RING) & 1u; }
  // the planes loaded at the start end here
  KFVM_RING_HD static int started(int k0, int last) { return k0 - 3 + RING < last ? k0 - 3 + RING : last; }
  // Where a wait gave up by plane k: the first and last plane whose load may still be in
  // flight.  A wait before the march ends it at plane k0, with every first plane in question;
  // a plane that landed, or was never asked for, costs no wait.
  KFVM_RING_HD static int flying_from(int k0, int k) { return k == k0 ? k0 - 2 : k; }
  KFVM_RING_HD static int flying_to(int k, int last) { return k + 2 < last ? k + 2 : last; }
};

} // namespace kfvm
