// fit_chain_kernel, wide layers, transposed rows of 32 node words.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_wide_rw32(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<32, true, true, false> : (const void *)fit_chain_kernel<32, true, false, false>;
    return hybrid ? (const void *)fit_chain_kernel<32, false, true, false> : (const void *)fit_chain_kernel<32, false, false, false>;
}
