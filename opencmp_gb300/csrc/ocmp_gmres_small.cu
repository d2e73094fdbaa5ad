// GMRES for queues of systems of few rows (ocmp_gmres.cuh): several blocks of 128 threads per SM, one
// system each.
#include "ocmp_gmres.cuh"

namespace ocmp {

template <>
const void* gm_small_kernel<double>() {
    return (const void*)gm_kernel<double, kGmSmallThreads>;
}
template <>
const void* gm_small_kernel<float>() {
    return (const void*)gm_kernel<float, kGmSmallThreads>;
}

}  // namespace ocmp
