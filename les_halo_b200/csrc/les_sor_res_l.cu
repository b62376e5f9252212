// les_sor_res_l.cu -- the chip-resident SOR kernel for 48 and 64 planes per
// thread (les_sor_res.cu).
#include <climits>

#include "les_press.cuh"
#include "les_sor_res.cuh"

const void *les_res_kernel_l(int seg) {
    using namespace les;
    return seg == 48 ? (const void *)k_sor_res<48, false> : (const void *)k_sor_res<64, true>;
}
