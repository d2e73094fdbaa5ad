// GMRES by teams of blocks that take one system after another from a queue (ocmp_gmres.cuh).
#include "ocmp_gmres.cuh"

namespace ocmp {

template <>
const void* gm_many_kernel<double>() {
    return (const void*)gm_kernel<double, kGmThreads<double>, true>;
}
template <>
const void* gm_many_kernel<float>() {
    return (const void*)gm_kernel<float, kGmThreads<float>, true>;
}

}  // namespace ocmp
