// fd3d_forms.cu -- the kernels of PML quotients that take a form of their own (PmlForm):
// a few per cent of spacings.  They stand in a module of their own because a program loads a whole
// module with the first of its kernels: in one with the others they made the first context of
// every process 5 ms later (32 ms instead of 27), the first batch 1.3 ms.
#include "fd3d_batch.cuh"
#include "fd3d_kernels.cuh"
#include "fd3d_opt.cuh"

namespace fd3d {

PmlKernel<float> pml_kernel_forms(bool stress, bool slab) {
    if (slab) return stress ? pml_kernel_of<float, true, true, true>() : pml_kernel_of<float, false, true, true>();
    return stress ? pml_kernel_of<float, true, false, true>() : pml_kernel_of<float, false, false, true>();
}
VelSmallKernel<float> vel_small_forms(bool layered) {
    return layered ? k_vel_small<float, true, true> : k_vel_small<float, false, true>;
}
StrSmallKernel<float> str_small_forms(bool layered) {
    return layered ? k_str_small<float, true, true> : k_str_small<float, false, true>;
}
BatchPmlKernel batch_pml_forms(bool stress) { return stress ? k_bpml<true, true> : k_bpml<false, true>; }
BatchHalfKernel batch_half_forms(bool stress) { return stress ? k_bhalf<true, true> : k_bhalf<false, true>; }

}  // namespace fd3d
