// Tile shapes of the air WENO sweeps and the choice of one for a block that was
// neither tuned nor set.  Host and device, no CUDA in it.
#pragma once

namespace cfk {

// nodes per column and columns per CTA, [0] x and [1] y/z sweeps
constexpr int kAirTileNodes[2][3] = {{63, 15, 31}, {31, 15, 7}};
constexpr int kAirTileColumns[2][3] = {{2, 8, 4}, {8, 16, 16}};

// The tile variant of sweep dir over ext nodes in columns of which `across` lie
// along the CTA's other axis and `outer` along the grid's: the shape whose
// tiles, cut to the multiples of both their sides, compute the fewest faces, a
// staged point counting a tenth of one.  us per sweep of the shapes and the
// choice: x (63x2, 15x8, 31x4), 161 nodes in 113 columns 247, 240, 250; 33 in 9
// (WENO5) 6.4, 7.9, 7.3; 17 in 200 89, 53, 52; 257 in 257 611, 586, 565.  y/z
// (31x8, 15x16), 97 nodes in 161 columns 291, 273; 113 in 161 258, 270; 64 in 17
// 60, 68; 257 in 257 2320, 2402 -- the smaller each time (49 x 130 x 20's y
// sweep, 33, 29, is one where it is not: 1.2 waves of CTAs).
// A sweep of one wave of CTAs (4 an SM) is as long as one CTA: there y and z
// take the 7x16 shape, whose faces are one round a thread instead of two
// (31x8, 15x16, 7x16; CTAs of 15x16): 32^3 (192) 14.6, 14.6, 10.5; 48^3 (576)
// 24.9, 24.1, 20.8; 33 x 65 x 33 (585) 26.9, 23.2, 20.7.  Beyond one wave it is
// as often behind: 52^3 (832) 28.9, 33.0, 31.0; 17 x 200 x 64 (1792) 49, 64, 62;
// 257 x 33 x 17 (867) 39.6, 33.1, 26.9; 64^3 (1280) 52.9, 45.4, 43.3.
inline int weno_air_tile(int ext, int across, int outer, int dir, int order, int n_sm) {
  const int yz = dir > 0, halo = order == 7 ? 8 : 6;
  if (yz && (long long)((across + 15) / 16) * ((ext + 14) / 15) * outer <= 4LL * n_sm) return 2;
  int best = -1;
  long long least = 0;
  for (int v = 0; v < (yz ? 2 : 3); ++v) {
    const int n = kAirTileNodes[yz][v], c = kAirTileColumns[yz][v];
    const long long cost =
        (long long)((ext + n - 1) / n) * ((across + c - 1) / c) * c * (10 * (n + 1) + n + halo);
    if (best < 0 || cost < least) {
      best = v;
      least = cost;
    }
  }
  return best;
}

}  // namespace cfk
