// k_coop_types.cu -- the whole-run kernel for several particle types.
#include "k_coop.cuh"

namespace femmd {

const void *coop_kernel_types(const DevSys &s) { return coop_image<true, false>(s); }

}  // namespace femmd
