// What an untuned launch of the tensor-core convolutions is expected to take, per tile shape: the choice among feature tiles of 64,
// 128 and 256, two or four epilogue groups, CTA pairs and the feature-row form.  The shape that keeps the device fullest per
// instruction (256 features) is the slowest one on a small grid: with a single tile per CTA the whole tile passes through one
// epilogue group, and most SMs have none.
//   time = launch + steps * step + epilogue + (waves - 1) * max(steps * step * overlap, epilogue of a tile in steady state)
// The constants (us) are a least-squares fit to 450 8-bit and 120 fp16 layers (those of ResNet-50, MobileNet-v2, AlexNet and VGG16
// and a few of none of them, 1 .. 256 images), every shape timed; on these same layers the shape with the lowest estimate is on average
// 3 % (8-bit) and 1 % (fp16) behind the fastest one, the fixed choice before (256 features wherever there are that many) 16 % and 29 %.
// The fp16 pairs came later: their two constants are set by hand from the pairs' timings.  On 345 fp16 layers outside the fit (1x1 and 3x3, 64
// .. 512 -> 128 .. 640 features at 13x13 .. 112x112, 1 .. 128 images) the choice is 2.2 % behind the fastest variant, at worst 65 %.
#pragma once
#include <algorithm>
#include <stdint.h>
#include "engine.hpp"

namespace b200 {

constexpr int64_t kCostSMs = 148;            // of the device the constants are fitted on (a choice is made without a device at hand)

enum TileKind { TILE_TWO_GROUPS = 0, TILE_FOUR_GROUPS = 1, TILE_PAIR = 2 };

struct TileCost {
    double launch, pair_launch;              // first load to last store of an empty tile; what a CTA pair adds
    double step, step_row, pair_step;        // a reduction step: fixed, per operand row of 128 bytes; factor in a pair
    double epi, epi_col, residual;           // latency of a tile's epilogue: fixed, per feature; factor with a fused residual
    double thr, thr_col, thr_col4;           // its share of the time in steady state, with two and with four groups
    double overlap;                          // main loop beside the epilogue of the tile before
};
constexpr TileCost kTileCostI8 = {3.37, 1.05, 0.218, 0.00016, 0.868, 1.31, 0.0082, 1.23, 0.33, 0.0065, 0.0048, 1.33};
constexpr TileCost kTileCostF16 = {3.19, 0.5, 0.240, 0.00024, 0.9, 1.09, 0.0100, 1.10, 0.40, 0.0078, 0.0078, 1.13};

// `m_tiles` tiles of 128 pixels, `steps` reduction steps of `bk` bytes
inline double tile_cost(const TileCost& c, int64_t m_tiles, int64_t ofm, int bn, int64_t steps, int bk, TileKind kind, bool fused)
{
    if (kind == TILE_PAIR) m_tiles = (m_tiles + 1) / 2 * 2;
    const int64_t n_tiles = (ofm + bn - 1) / bn, waves = (m_tiles * n_tiles + kCostSMs - 1) / kCostSMs;
    auto whole = [](int64_t v) { return (v + 63) / 64 * 64; };
    const double widest = (double)(n_tiles == 1 ? std::min<int64_t>(bn, whole(ofm)) : bn);
    const double typical = (double)std::min<int64_t>(bn, whole((ofm + n_tiles - 1) / n_tiles));
    const double main = (double)steps * (c.step + c.step_row * (128 + bn) * (bk / 128.0)) * (kind == TILE_PAIR ? c.pair_step : 1.0);
    const double res = fused ? c.residual : 1.0;
    const double epi = (c.epi + c.epi_col * widest) * res;
    const double thr = (c.thr + (kind == TILE_FOUR_GROUPS ? c.thr_col4 : c.thr_col) * typical) * res;
    return c.launch + (kind == TILE_PAIR ? c.pair_launch : 0.0) + main + epi + (double)(waves - 1) * std::max(main * c.overlap, thr);
}

}  // namespace b200
