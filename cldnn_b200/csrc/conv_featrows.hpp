// The feature-row form of the tensor-core convolutions (conv_featrows.cu), reached through tuning indices of conv_i8_tc and
// conv_f16_tc: few output pixels, long reductions, inner products.
#pragma once
#include <string>
#include "engine.hpp"

namespace b200 {

struct FrPlan {
    int mode;                                // 0 flat, 1 TMA im2col, 2 tiled box (over pixels)
    int cols, split;                         // pixel columns per tile, CTAs that share a tile's reduction
    int bw, bh, bb;                          // tiled: box of pixels
};

constexpr int kFrCols = 5;                   // 16, 32, 64, 128, 256 pixel columns
constexpr int kFrSplits = 4;                 // 1, 2, 4, 8 CTAs per tile
constexpr int kFrVariants = kFrCols * kFrSplits;

// variant 0 .. kFrVariants - 1 = columns index * 4 + split index.  `p` has passed the layout checks of the calling kernel's plan.
bool fr_plan(const cldnn_b200_conv_params& p, int variant, FrPlan& pl, std::string* why);
// The variant an untuned inner product (a pointwise convolution of 1x1 maps) takes; -1: the pixel-row kernels are the better choice.
int fr_inner_product_variant(const cldnn_b200_conv_params& p);
// The variant with the lowest expected time (us, returned) for a convolution of any shape, among those whose CTAs are
// all resident at once; -1: none.
double fr_cost(const cldnn_b200_conv_params& p, int& variant);
int32_t fr_prepare(cldnn_b200_ctx_impl* ctx, const cldnn_b200_conv_params& p, const cldnn_b200_args* a, const FrPlan& pl, cldnn_b200_prepared_impl* out);

}  // namespace b200
