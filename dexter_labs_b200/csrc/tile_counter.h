// The counter of a tile that several CTAs share: all but one park their sums in global scratch, the last
// one waits for them and finishes the tile.  Low half: sums parked; high half: CTAs that are through with
// the tile, whether they parked, finished or gave up on a wait.  Whoever is last to leave sets it back
// to zero, so that a launch after one that ran into a wait's limit starts clean, whichever CTA gave up and
// in whatever order they leave.  In a launch that runs through that is the finisher, which knows
// that the others have left and stores the zero without counting itself.
#pragma once

#ifdef __CUDACC__
#define DX_HD __host__ __device__ __forceinline__
#else
#define DX_HD inline
#endif

namespace dx {
constexpr unsigned kTileParked = 1u, kTileLeft = 1u << 16;

// What a leaving CTA adds.
DX_HD unsigned tile_leave_add(bool parked) { return kTileLeft + (parked ? kTileParked : 0u); }
// `before`: the counter before that; true for the last of `sharers` CTAs.
DX_HD bool tile_all_left(unsigned before, int sharers) { return static_cast<int>(before >> 16) + 1 == sharers; }
// What the finisher waits for.
DX_HD bool tile_all_parked(unsigned now, int sharers) { return static_cast<int>(now & 0xFFFFu) == sharers - 1; }
}  // namespace dx
