// k_coop_sigma.cu -- the whole-run kernel for a sigma per particle.
#include "k_coop.cuh"

namespace femmd {

const void *coop_kernel_sigma(const DevSys &s) {
    return s.numTypes > 1 ? coop_image<true, true>(s) : coop_image<false, true>(s);
}

}  // namespace femmd
