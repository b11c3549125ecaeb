// rd_tile_rule.hpp -- which tiles of a fused tiled run whole clusters evolve, and which
// of their keys are folded in segments.
#pragma once

#include <algorithm>
#include <cstdint>

namespace rdb {

// Process-wide settings as the caller gave them; 0 leaves a threshold to tile_rule.
struct TileClusterParams {
    bool enabled = true;
    int min_points = 0;   // evolve points from which a whole cluster evolves a tile
    int seg_min = 0;      // members from which it folds a key in segments
};

// what a caller who left a threshold to the rule is told it is: the rule never goes
// above the first, and its second is 12,288 (TILE_SEG_RULE)
constexpr int TCL_MIN_POINTS = 100000, TSEG_MIN = 8192;
// below this one CTA's passes are shorter than the cluster's barriers
constexpr int TCL_SMALLEST = 4096;
constexpr int TILE_SEG_RULE = 12288;

struct TileRule {
    int64_t heavy;        // evolve points from which a tile is heavy
    int seg_min;
    bool clusters;        // the cluster kernel runs (it evolves light tiles too)
    bool hand_over;       // and its CTAs hand over light tiles at the end
};

// A caller's threshold holds as it is.  Left to the rule, a tile is heavy from a
// 4 x SMs-th of all evolve points on (half of what each of the resident CTAs would
// get): a larger one evolved by one CTA outlasts the other tiles.  And a key is
// folded in segments from 12,288 members on, not 8,192: where its coordinates lie on
// both sides of zero the segments' runs break at every change of binade, and one
// warp's add chain is faster.  Whole solves, ms, thresholds of 100,000 points and
// 8,192 members / these rules with the hand-over of rd_tile_cluster.cuh: 1M spiral
// in 70 leaves 190 / 35, in 1,024 tiles 46 / 18, 2M in 582 leaves 69 / 32, 300,000
// in 256 tiles 48 / 17; the 10M spiral in 4,096 tiles keeps its 100,000 (34.9 / 32.7;
// 48 with 10,000).
inline TileRule tile_rule(const TileClusterParams& p, int64_t total_points, int sms, int64_t largest_tile)
{
    const bool by_rule = p.min_points <= 0;
    TileRule r;
    r.heavy = by_rule ? std::min<int64_t>(TCL_MIN_POINTS, std::max<int64_t>(TCL_SMALLEST, total_points / (4 * sms)))
                      : p.min_points;
    r.seg_min = p.seg_min > 0 ? p.seg_min : TILE_SEG_RULE;
    r.hand_over = p.enabled && by_rule && largest_tile >= TCL_SMALLEST;
    r.clusters = p.enabled && (r.hand_over || largest_tile >= r.heavy);
    return r;
}

}  // namespace rdb
