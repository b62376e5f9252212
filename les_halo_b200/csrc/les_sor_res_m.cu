// les_sor_res_m.cu -- the chip-resident SOR kernel for 32 and 40 planes per
// thread (les_sor_res.cu).
#include <climits>

#include "les_press.cuh"
#include "les_sor_res.cuh"

const void *les_res_kernel_m(int seg) {
    using namespace les;
    return seg == 32 ? (const void *)k_sor_res<32, false> : (const void *)k_sor_res<40, false>;
}
