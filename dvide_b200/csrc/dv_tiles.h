// dv_tiles.h -- which tiles of a scene a member of its team takes, in host and
// device code.
//
// The passes that copy contacts ahead walk the contact tiles alone; the others
// walk all tiles, the contacts' and then the bilateral rows'.  Both walks give a
// member the same contact tiles in the same order, in every launch shape: what
// one pass leaves in a member's stages or in L2 is what the other asks for.
#pragma once

#ifndef DV_HD
#ifdef __CUDACC__
#define DV_HD __host__ __device__
#else
#define DV_HD
#endif
#endif

namespace dv {

struct TileShare {
  int rank, m;            // the member's place among the team's m
  int chunk, contiguous;  // round robin in chunks of `chunk` tiles, or one range per member
};

// Tile i of the member's share of n tiles; -1 past the end.
DV_HD inline int share_tile(const TileShare& t, int n, int i) {
  if (t.contiguous) {
    const int lo = (int)((long long)n * t.rank / t.m);
    const int hi = (int)((long long)n * (t.rank + 1) / t.m);
    return lo + i < hi ? lo + i : -1;
  }
  const int k = t.chunk;
  const int x = k == 1 ? t.rank + i * t.m : (t.rank + (i / k) * t.m) * k + i % k;
  return x < n ? x : -1;
}

// Tile i of the member's share of a scene whose first ntc tiles of nt are the
// contacts'.  Round robin deals all of them at once; ranges are cut from the
// contacts' tiles and from the rows' apart.
DV_HD inline int scene_tile(const TileShare& t, int ntc, int nt, int i) {
  if (!t.contiguous || nt == ntc) return share_tile(t, nt, i);
  const int lo = (int)((long long)ntc * t.rank / t.m);
  const int hi = (int)((long long)ntc * (t.rank + 1) / t.m);
  if (i < hi - lo) return lo + i;
  const int x = share_tile(t, nt - ntc, i - (hi - lo));
  return x < 0 ? -1 : ntc + x;
}

}  // namespace dv
