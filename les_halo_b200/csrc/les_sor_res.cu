// les_sor_res.cu -- the chip-resident SOR kernel's instantiations, one
// translation unit per few of them: each unrolls a segment's planes, so they
// are the slowest part of the build.
#include <climits>

#include "les_press.cuh"
#include "les_sor_res.cuh"

const void *les_res_kernel_m(int seg);  // les_sor_res_m.cu: 32, 40
const void *les_res_kernel_l(int seg);  // les_sor_res_l.cu: 48, 64

// The kernel of SEG planes per thread (nullptr: none).
const void *les_res_kernel(int seg) {
    using namespace les;
    switch (seg) {
        case 8: return (const void *)k_sor_res<8, false>;
        case 16: return (const void *)k_sor_res<16, false>;
        case 24: return (const void *)k_sor_res<24, false>;
        case 32:
        case 40: return les_res_kernel_m(seg);
        case 48:
        case 64: return les_res_kernel_l(seg);
    }
    return nullptr;
}
