// k_coop_fast.cu -- the whole-run kernel in the fast force mode (sigma by type).
#include "k_coop.cuh"

namespace femmd {

const void *coop_kernel_fast(const DevSys &s) {
    return s.numTypes > 1 ? coop_image<true, false, true>(s) : coop_image<false, false, true>(s);
}

}  // namespace femmd
