// fit_chain_kernel for transposed rows of 16 node words.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_rw16(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<16, true, true> : (const void *)fit_chain_kernel<16, true, false>;
    return hybrid ? (const void *)fit_chain_kernel<16, false, true> : (const void *)fit_chain_kernel<16, false, false>;
}
