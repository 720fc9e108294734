// fit_chain_kernel, narrow layers, transposed rows of 16 node words.
#include "gtm_fit_chain.cuh"

const void *fit_chain_kernel_narrow_rw16(bool one_layer, bool hybrid)
{
    using namespace gtm;
    if (one_layer) return hybrid ? (const void *)fit_chain_kernel<16, true, true, true> : (const void *)fit_chain_kernel<16, true, false, true>;
    return hybrid ? (const void *)fit_chain_kernel<16, false, true, true> : (const void *)fit_chain_kernel<16, false, false, true>;
}
