// Geometry of a 2-D convolution, shared by the unfolding path (om_spatial.cu), the kernels of om_conv_tc.cu and om_conv_fma.cu.
#pragma once
#include "om_common.cuh"

namespace om {

struct ConvGeom {
  int n, cin, h, w, cout, kh, kw, sh, sw, pt, pl, dh, dw, groups, oh, ow;
};

// The TF32 products without an unfolded matrix (om_conv_tc.cu). *_fits says whether the kernel takes the geometry; the caller
// has already decided that the product runs on the tensor pipe.
bool conv_tc_fwd_fits(const ConvGeom& g);
int32_t conv_tc_fwd(om_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y);
bool conv_tc_wgrad_fits(const ConvGeom& g);
int32_t conv_tc_wgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* x, float* dw, int accumulate);

// The same from channels-last copies of the activations, for the geometries whose pixels and channels tile well.
bool conv_nhwc_fwd_fits(const ConvGeom& g);
int32_t conv_nhwc_fwd(om_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y);
bool conv_nhwc_dgrad_fits(const ConvGeom& g);
int32_t conv_nhwc_dgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* w, float* dx, const float* turned_gr = nullptr);
bool conv_nhwc_wgrad_fits(const ConvGeom& g);
int32_t conv_nhwc_wgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* x, float* dw, int accumulate, const float* turned_gr = nullptr);
// The channels-last copy of the output's gradient that weight and input gradient take (turned_gr above): its floats, and the pass that writes it and, when asked
// for, the bias gradient.
long long conv_nhwc_turned_floats(const ConvGeom& g);
int32_t conv_nhwc_turn_gradient(om_ctx* ctx, const ConvGeom& g, const float* gr, float* turned, float* dbias, int accumulate_b);

// The fp32 products of small shapes without an unfolded matrix (om_conv_fma.cu).
bool conv_fma_fwd_fits(const ConvGeom& g);
int32_t conv_fma_fwd(om_ctx* ctx, const ConvGeom& g, const float* x, const float* w, const float* bias, float* y);
bool conv_fma_dgrad_fits(const ConvGeom& g);
int32_t conv_fma_dgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* w, float* dx);
bool conv_fma_wgrad_fits(const ConvGeom& g);
int32_t conv_fma_wgrad(om_ctx* ctx, const ConvGeom& g, const float* gr, const float* x, float* dw, int accumulate);

}  // namespace om
