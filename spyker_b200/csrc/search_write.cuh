#pragma once

#include "common.cuh"

namespace spk
{
// Spikes (and pooled spikes) of a search layer from its per-pixel records;
// see search_write.cu.  `codes`: scratch of 16 bytes per pixel (used for maps
// above 16384 pixels only).
struct SearchWrite
{
    const int4 *records;  // [b * oh * ow]: (winning channel, first step, ...)
    uint8_t *codes;
    const int *negw, *flag;  // off the search path when either is set
    uint8_t *spikes, *pooled;  // pooled: null for none
    int64_t b;
    int T, C, oh, ow, pky, pkx, poh, pow_;
};

void search_write(const SearchWrite &W, cudaStream_t s);
}  // namespace spk
