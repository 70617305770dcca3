// site_terms.cuh: what a launch of the assembly's site pass takes (k_site_terms, site_terms.cu).
#pragma once

#include "device.cuh"

namespace nb
{

struct SiteArgs
{
    void* terms;                        // [site][c] over every plane: doubles, or floats (MIXED)
    float4* y;                          // [site]: the site's sample of the other latent
    const float* tgt;                   // [fractional site][NOUT]: the targets of the sites j > 0 (k_site_targets)
    long long site0[MAX_PLANES + 1];    // the first site of each plane in `terms`
    long long tsite0[MAX_PLANES + 1];   // the first fractional site of each plane in `tgt`
    unsigned span;                      // pixels of one block
};

// Every plane's sites: the gradient terms and the other latent's samples (MIXED: FP32 terms). One module per output count
// and form (site_terms.cu).
template <int NOUT, bool MIXED>
void launch_site_terms(const nntc_b200_device* d, const Planes& S, SiteArgs A, int level0, cudaStream_t stream);

}   // namespace nb
