// fit_chain_kernel, narrow layers, transposed rows of 1 node word.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_narrow_rw1(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<1, true, true, true> : (const void *)fit_chain_kernel<1, true, false, true>;
    return hybrid ? (const void *)fit_chain_kernel<1, false, true, true> : (const void *)fit_chain_kernel<1, false, false, true>;
}
