// Internal interface of the U-Net denoiser's kernels (unet_kernels.cu,
// unet_tc.cu) for the network code (unet.cpp).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace unet {

struct ConvShape {
    int B, H, W, Cin, Cout;
};

// out[.., out_offset + co] (row stride out_stride) = act(bias + conv3x3(in, w)), padding 1.
cudaError_t conv_fwd(const ConvShape& s, const void* in, bool in_f32, const __nv_bfloat16* w, const float* bias,
                     bool relu, void* out, bool out_f32, int out_stride, int out_offset, cudaStream_t st);
// dw += d loss / d w, db += d loss / d bias, from the layer input and the gradient of its output.
cudaError_t conv_wgrad(const ConvShape& s, const __nv_bfloat16* in, const float* dout, float* dw, float* db,
                       cudaStream_t st);
// Gradient through a ReLU: g = 0 where its output y is not positive.
cudaError_t relu_grad(long n, const __nv_bfloat16* y, float* g, cudaStream_t st);
cudaError_t pool_fwd(int B, int H, int W, int C, const __nv_bfloat16* in, __nv_bfloat16* out, cudaStream_t st);
cudaError_t pool_bwd(int B, int H, int W, int C, const __nv_bfloat16* in, const __nv_bfloat16* out,
                     const float* gout, float* gin, cudaStream_t st);
cudaError_t up_fwd(int B, int h, int w, int C, const __nv_bfloat16* in, __nv_bfloat16* out, int stride, int offset,
                   cudaStream_t st);
cudaError_t up_bwd(int B, int h, int w, int C, const float* gout, int stride, int offset, float* gin,
                   cudaStream_t st);
cudaError_t copy_channels(long pixels, int C, const __nv_bfloat16* src, __nv_bfloat16* dst, int stride, int offset,
                          cudaStream_t st);
cudaError_t add_channels(long pixels, int C, const float* src, int stride, int offset, float* dst, cudaStream_t st);
cudaError_t make_input(long pixels, const float* src, __nv_bfloat16* dst, int stride, cudaStream_t st);
cudaError_t frame_input(int W, int H, int Wp, int Hp, const float* color, const float* aux7, const float* depth,
                        __nv_bfloat16* dst, int stride, cudaStream_t st);
cudaError_t frame_output(int W, int H, int Wp, int stride, const float* pred, float* out, cudaStream_t st);
cudaError_t l1_loss(long pixels, int stride, const float* pred, const float* target, float* grad, float* loss,
                    cudaStream_t st);
// The fused steps of the tensor-core backward. Each leaves the gradient at an
// activation, masked by its ReLU and rounded to bf16, in g16 (the operand of
// the next weight and input gradients), and adds the masked float gradient's
// sum over pixels to db, the bias gradient of the layer that made it.
//
// l1_back: l1_loss, the gradient as float4 per pixel (g4, channels past the
// third are zero) and in 16 bf16 channels (g16), and the sums (db).
cudaError_t l1_back(long pixels, const float* pred, const float* target, float4* g4, __nv_bfloat16* g16, float* db,
                    float* loss, cudaStream_t st);
// last_back: through the last layer (wt [32][9][16] flip-transposed) to its
// input y (32 channels), in float from g4's three channels.
cudaError_t last_back(int B, int H, int W, const float4* g4, const __nv_bfloat16* wt, const __nv_bfloat16* y,
                      __nv_bfloat16* g16, float* db, cudaStream_t st);
// up_back: through the 2x upsampling whose output is channels [0, C) of gcat
// (stride channels, 2h x 2w) to y (h x w, C channels).
cudaError_t up_back(int B, int h, int w, int C, const float* gcat, int stride, const __nv_bfloat16* y,
                    __nv_bfloat16* g16, float* db, cudaStream_t st);
// skip_back: the gradient at y (H x W, C channels) from its copy in channels
// [offset, offset + C) of gcat and through its 2x2 max pool.
cudaError_t skip_back(int B, int H, int W, int C, const float* gcat, int stride, int offset, const __nv_bfloat16* y,
                      const __nv_bfloat16* pooled, const float* gpool, __nv_bfloat16* g16, float* db, cudaStream_t st);
// w_t[ci][tap][co] = w[co][8 - tap][ci] of every layer: the weights of the
// transposed convolutions that carry gradients back to a layer's input.
struct FlipLayers {
    int n, cin[16], cout[16];
    long off[16];
};
cudaError_t flip_transpose_all(const FlipLayers& layers, const __nv_bfloat16* w, __nv_bfloat16* wt, cudaStream_t st);
cudaError_t make_output(long pixels, int stride, const float* pred, float* out, cudaStream_t st);
cudaError_t adam(long n, float* w, const float* g, float* m, float* v, __nv_bfloat16* w16, float lr, int step,
                 cudaStream_t st);
cudaError_t f32_to_bf16(long n, const float* a, __nv_bfloat16* b, cudaStream_t st);

// Where the tensor-core convolution writes its result (any pointer may be
// null): out[p * stride + offset + co] (bf16, or float for out_f32); a bf16
// copy into out2 at the same pixel, or (up2) at the four pixels of the 2x
// finer level it covers -- the halves of a decoder's concatenation; and the
// 2x2 max pool of the result into pool ([pixel][Cout], bf16).
struct ConvOut {
    void* out = nullptr;
    int stride = 0, offset = 0;
    __nv_bfloat16* out2 = nullptr;
    int stride2 = 0, offset2 = 0, up2 = 0;
    __nv_bfloat16* pool = nullptr;
    // Backward: the result is kept where mask ([pixel][Cout], bf16) is
    // positive and zero elsewhere, and its sum over pixels is added to
    // colsum (Cout floats). bf16 output, Cout a multiple of 32.
    const __nv_bfloat16* mask = nullptr;
    float* colsum = nullptr;
    // The network's last layer: the first three channels as radiance, 3
    // floats per pixel of an image of image_w x image_h per batch entry (the
    // part of the padded frame that the caller asked for).
    float* image = nullptr;
    int image_w = 0, image_h = 0;
};

// Tensor-core forward convolution (tcgen05, accumulators in TMEM). Returns
// cudaErrorNotSupported for shapes it does not take (Cin % 32, Cout % 16 or
// Cout > 256; odd sizes with pool), which then run on conv_fwd.
cudaError_t conv_fwd_tc(const ConvShape& s, const __nv_bfloat16* in, const __nv_bfloat16* w, const float* bias,
                        bool relu, const ConvOut& o, bool out_f32, unsigned int* status, cudaStream_t st);

// Tensor-core weight gradient (tcgen05, MN-major operands): dw += d loss /
// d w from the layer input and the bf16 gradient of its output (Cout <= 128, a
// multiple of 8, Cin a multiple of 32), float atomics. cudaErrorNotSupported
// for other shapes, which then run on conv_wgrad.
cudaError_t conv_wgrad_tc(const ConvShape& s, const __nv_bfloat16* in, const __nv_bfloat16* dout, float* dw,
                          unsigned int* status, cudaStream_t st);

}  // namespace unet
