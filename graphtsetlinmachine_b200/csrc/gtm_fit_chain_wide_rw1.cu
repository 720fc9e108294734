// fit_chain_kernel, wide layers, transposed rows of 1 node word.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_wide_rw1(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<1, true, true, false> : (const void *)fit_chain_kernel<1, true, false, false>;
    return hybrid ? (const void *)fit_chain_kernel<1, false, true, false> : (const void *)fit_chain_kernel<1, false, false, false>;
}
