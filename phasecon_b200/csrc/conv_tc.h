// The U-Net's convolutions on the fifth-generation tensor cores (unet_tc.cu).
#pragma once
#include <cstddef>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace mbirgpu {

// One convolution's weights in the parameter array (w, elements) and where their
// re-laid forward and data-gradient forms go (elements); nt, nt_grad: output
// channels per CTA of each (conv_tc_split), 0 where the tensor-core kernel does
// not serve the shape.
struct ConvTcWeights {
    int cin, cout, nt, nt_grad;
    size_t w, out, out_grad;
};
// A convolution's input: channels 0 .. ca - 1 from a, the rest from b (the decoder's
// concatenation), both [voxel][channel]; up: a is on the grid of half the size and
// read by nearest upsampling. Reading it in place saves writing and reading the
// concatenated and the upsampled tensors (0.9 of 22 ms of a warm start's 8 frames).
struct ConvIn {
    const __nv_bfloat16 *a, *b;
    int ca, cb, up;

    // the 8 channels from ch on of voxel (z, y, x) of the h x w grid
    __device__ __forceinline__ const __nv_bfloat16 *piece(int z, int y, int x, int h, int w, int ch) const
    {
        const bool second = ch >= ca;
        const long long v = up ? ((long long)(z >> 1) * (h >> 1) + (y >> 1)) * (w >> 1) + (x >> 1)
                               : ((long long)z * h + y) * w + x;
        return second ? b + v * cb + (ch - ca) : a + v * ca + ch;
    }
};
int conv_tc_split(int Kin, int Nout);
// whether the tensor-core kernel serves the shape and the grid
bool conv_tc_serves(int Kin, int Nout, int d, int df);
void conv_tc_weights(const ConvTcWeights *list, int n, const __nv_bfloat16 *params, __nv_bfloat16 *out, cudaStream_t st);
int conv_tc_launch(const ConvIn &in, int Kin, const __nv_bfloat16 *wtc, const float *bias, __nv_bfloat16 *out,
                   int Nout, int d, int h, int w, int df, int relu, cudaStream_t st);
int conv_tc_status(cudaStream_t st);

}  // namespace mbirgpu
