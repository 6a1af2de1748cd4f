// The feature-row form of the tensor-core convolutions (conv_featrows.cu), reached through tuning indices of conv_i8_tc and
// conv_f16_tc: few output pixels, long reductions, inner products.
#pragma once
#include <string>
#include "engine.hpp"

namespace b200 {

// A convolution in groups as the tensor-core kernels see it: every feature tile of 128 lies inside one group and reads that group's
// slice of the input features (a channel offset of the activation copies), with weights that hold the group's features only, zero
// padded to whole chunks of the reduction.  A chunk that reaches past the slice meets the padding's zeros, which is enough for integers;
// in fp16 zero times an Inf or NaN of the next group would be NaN, so there each group gets a tensor map that ends with its slice (zeros
// come in behind it), for up to kGroupMaps groups.  `p` comes in with feature counts per group and leaves with all output features in
// `ofm`; `ifm` stays the reduction's.
constexpr int kGroupMaps = 4;
inline int64_t chunk_bytes(int64_t cs) { return cs % 128 == 0 ? 128 : (cs % 64 == 0 ? 64 : 32); }   // of a tap's `cs` stored bytes
inline bool slices_overhang(const cldnn_b200_conv_params& p) { return p.groups > 1 && p.in.dtype == CLDNN_B200_F16 && p.ifm * 2 % chunk_bytes(p.w_px * 2); }
inline bool grouped_view(cldnn_b200_conv_params& p, std::string* why)
{
    auto no = [&](const char* m) { if (why) *why = m; return false; };
    if (p.groups == 1) return true;
    const int64_t es = p.in.dtype == CLDNN_B200_F16 ? 2 : 1;
    if (p.groups < 1 || p.fused_eltw) return no("grouped convolution: no fused residual");
    if (p.ofm < 128 || p.ofm % 128 || p.ifm * es % 16) return no("grouped convolution: whole feature tiles of 128 and 16-byte slices per group");
    if (p.w_px * es % 32 || p.w_px < p.ifm || p.w_px * es >= p.ifm * es + 128) return no("grouped convolution: weights must hold one group's features, padded to whole chunks");
    if (p.groups > kGroupMaps && slices_overhang(p)) return no("grouped fp16 convolution: slices of more than four groups must be whole chunks of the reduction");
    p.ofm *= p.groups;
    return true;
}
inline int64_t reduction_features(const cldnn_b200_conv_params& p) { return p.groups == 1 ? p.in.px : p.w_px; }   // stored, per tap

struct FrPlan {
    int mode;                                // 0 flat, 1 TMA im2col, 2 tiled box (over pixels)
    int cols, split;                         // pixel columns per tile, CTAs that share a tile's reduction
    int bw, bh, bb;                          // tiled: box of pixels
};

constexpr int kFrCols = 5;                   // 16, 32, 64, 128, 256 pixel columns
constexpr int kFrSplits = 4;                 // 1, 2, 4, 8 CTAs per tile
constexpr int kFrVariants = kFrCols * kFrSplits;

// variant 0 .. kFrVariants - 1 = columns index * 4 + split index.  `p` has passed the layout checks of the calling kernel's plan.
// `box`: also choose the tiled mode's box (a search over the map; whether the variant fits does not depend on it).
bool fr_plan(const cldnn_b200_conv_params& p, int variant, FrPlan& pl, std::string* why, bool box = true);
// The variant an untuned inner product (a pointwise convolution of 1x1 maps) takes; -1: the pixel-row kernels are the better choice.
int fr_inner_product_variant(const cldnn_b200_conv_params& p);
// The variant with the lowest expected time (us, returned) for a convolution of any shape, among those whose CTAs are
// all resident at once; -1: none.
double fr_cost(const cldnn_b200_conv_params& p, int& variant);
int32_t fr_prepare(cldnn_b200_ctx_impl* ctx, const cldnn_b200_conv_params& p, const cldnn_b200_args* a, const FrPlan& pl, cldnn_b200_prepared_impl* out);

}  // namespace b200
