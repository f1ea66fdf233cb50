// k_coop_slot.cu -- the fast mode's whole-run kernel (k_coop.cuh) with the
// energies grouped by storage slot: small systems of one type (coop_by_slot).
// Kernels of their own: branches for it in the others cost 144 disks in solvent
// 2 % (2130 -> 2177 us a run(100)).
#include "k_coop.cuh"

namespace femmd {

const void *coop_kernel_slot(const DevSys &s) { return coop_image<false, false, true, true>(s); }

}  // namespace femmd
