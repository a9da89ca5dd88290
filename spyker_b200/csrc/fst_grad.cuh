#pragma once

#include "common.cuh"

namespace spk
{
// Gradients of a first-spike conv layer from the non-zero output gradients;
// see fst_grad.cu.
struct FstGrad
{
    const float *t_in, *kernel, *t_out, *grad_out;
    int64_t b;
    int cin, h, w, cout, kh, kw, oh, ow, sy, sx, top, left, bottom, right;
};

// Partial sums of the kernel gradient: at least `least` sample groups, more
// (to fill the chip) within 64 MB.
int64_t fst_grad_w_groups(int64_t b, int64_t weights, int64_t least);
// Returns false, having done nothing, where the layer does not fit or the other
// kernel, of about general_us, is the faster.
bool fst_grad_in(const FstGrad &F, float *grad_in, double general_us, cudaStream_t s);
// part: [groups][cout * cin * kh * kw] FP64 sums over consecutive samples;
// returns the groups written, 0 (having done nothing) where the layer does
// not fit.
int64_t fst_grad_w(const FstGrad &F, double *part, int64_t groups, cudaStream_t s);
}  // namespace spk
