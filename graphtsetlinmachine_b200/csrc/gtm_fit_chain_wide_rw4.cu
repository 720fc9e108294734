// fit_chain_kernel, wide layers, transposed rows of 4 node words.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_wide_rw4(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<4, true, true, false> : (const void *)fit_chain_kernel<4, true, false, false>;
    return hybrid ? (const void *)fit_chain_kernel<4, false, true, false> : (const void *)fit_chain_kernel<4, false, false, false>;
}
