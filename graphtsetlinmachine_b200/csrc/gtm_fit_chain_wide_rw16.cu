// fit_chain_kernel, wide layers, transposed rows of 16 node words.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_wide_rw16(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<16, true, true, false> : (const void *)fit_chain_kernel<16, true, false, false>;
    return hybrid ? (const void *)fit_chain_kernel<16, false, true, false> : (const void *)fit_chain_kernel<16, false, false, false>;
}
