// Grids of the fully-sharded collectives. Each rank of a launch has `groups` groups (destinations, owners) of `tiles` tiles.
#pragma once
#include <algorithm>
#include <cstdint>

namespace nangila {

// A CTA for every tile (x) of every group (y); or, where the caller allows a rank fewer CTAs (`cap` above 0), as many of them for each group as that leaves,
// which walk the group's tiles in steps of x; with fewer CTAs than groups one for each of y groups, in steps of y. (Tiles of all groups
// numbered through and dealt out to all CTAs: 10 to 16 % slower for 4 x 6.3 M elements and 148 CTAs, since all of them work for one group at a time.)
enum Walk { kNoWalk, kWalkTiles, kWalkGroups };  // what a CTA does: one tile; tiles of its group; those of several groups
struct FsdpGrid {
  unsigned x, y;
  Walk walk;
};
inline FsdpGrid fsdp_grid(int64_t tiles, int groups, int cap) {
  tiles = std::max<int64_t>(1, tiles);
  groups = std::max(1, groups);
  if (cap <= 0 || int64_t(cap) >= tiles * groups) return {unsigned(tiles), unsigned(groups), kNoWalk};
  if (cap < groups) return {1u, unsigned(cap), kWalkGroups};
  return {unsigned(std::min<int64_t>(tiles, cap / groups)), unsigned(groups), kWalkTiles};
}
constexpr int64_t kMaxTiles = 0x3fffffff;  // of a group: a CTA counts them in 32 bits

}  // namespace nangila
