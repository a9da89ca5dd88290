#pragma once

#include "common.cuh"

namespace spk
{
// First-spike layer forward by walking each output pixel's inputs in spike
// order; see fst_walk.cu.
struct FstWalk
{
    const float *t_in;    // [b, cin, h, w]
    const float *kernel;  // [cout, cin, kh, kw]
    float *t_out;         // [b, cout, oh, ow]
    int64_t b;
    int cin, h, w, cout, kh, kw, sy, sx, top, left, oh, ow, time;
    float threshold;
    int terms;  // BF16 terms per weight (2 or 3)
};

// Bytes of scratch, 0 where the walk does not apply.
size_t fst_walk_workspace(int64_t b, int64_t cin, int64_t h, int64_t w, int64_t cout, int64_t kh, int64_t kw);
// Whether it is the faster one of the two forms (the dense kernel's: conv_tc.cu).
bool fst_walk_pays(int64_t npix, int64_t cin, int64_t taps, int64_t cout, int64_t time);
void fst_walk(const FstWalk &F, void *ws, cudaStream_t s);
}  // namespace spk
