// attention_span.h -- where the partial results of an evenly dealt decode step lie (attention.cu; no CUDA needed).
//
// Each CTA has two places: 2 cta for the item in which its share begins, 2 cta + 1 for the one that begins in its share.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LUX_HOST_DEVICE __host__ __device__
#else
#define LUX_HOST_DEVICE
#endif

namespace luxcuda {

// An item (a sequence's KV head): the CTA in which it begins and how many work on it.
struct AttnSpan {
    int32_t first, ctas;
};

// Whether the merge may follow it.  A CTA whose bounded wait gave up has not written the spans of the items that begin in its
// share: what is read then is whatever the scratch held.
LUX_HOST_DEVICE constexpr bool span_fits(AttnSpan s, uint32_t grid) {
    return s.first >= 0 && s.ctas >= 1 && (uint32_t)s.first < grid && (uint32_t)s.ctas <= grid - (uint32_t)s.first;
}
// The place of the item's partial result i < ctas.
LUX_HOST_DEVICE constexpr uint32_t span_place(AttnSpan s, uint32_t i) {
    return i == 0 ? 2u * (uint32_t)s.first + 1u : 2u * ((uint32_t)s.first + i);
}

}  // namespace luxcuda
