// How the FP32 source-location kernel is laid out (distributions.cu): a rule on sizes
// alone, so that it can be checked without a GPU.
#pragma once

#include <cstdint>

namespace hmc {

constexpr int SL_BY = 8;  // event lanes per block at most

struct SrclocShape {
  int lanes;   // events of a block at a time
  int blocks;  // of a cluster, which share a tile's events
};

// One cluster per tile of 32 chains, a block for every eight events up to eight, so that
// few chains still fill the chip.  Where the tiles fill it (four blocks on an SM) and
// the stations are few, staging them and the cluster's two barriers cost more than the
// idle lanes of a loop over events: fewer blocks then, one from 28 800 chains on.  On a
// full chip, events that leave a fifth of the lanes idle (a sixth, counting the rounds
// of fewer blocks) are spread evenly over them, as nine events in two blocks of eight
// lanes leave one block waiting for the other; elsewhere all eight lanes help to stage
// the stations.  Misfits: 64 events, 4 stations, 30 000 chains 20.5
// us with one block and 48.2 with eight; 9 events, 700 stations, 30 000 chains 124 us
// with even lanes and 180 with eight; 33 events, 200 stations, 2500 chains 16.5 us with
// five blocks and 32.5 with one.
inline SrclocShape srcloc_shape(int64_t E, int64_t S, int64_t C) {
  const int64_t groups = (E + SL_BY - 1) / SL_BY, tiles = (C + 31) / 32;
  int most = 8;
  if (tiles >= 2048 || (tiles >= 900 && S < 100))
    most = 1;
  else if (S < 30)
    while (most > 1 && (groups < most ? groups : most) * tiles > 4 * 152) --most;
  SrclocShape s{SL_BY, groups < most ? (int)groups : most};
  if (E > SL_BY && tiles * s.blocks > 152) {
    const int64_t slots = (groups + s.blocks - 1) / s.blocks * s.blocks;
    const bool idle = most < 8 ? 6 * (slots * SL_BY - E) >= slots * SL_BY : 5 * (groups * SL_BY - E) >= groups * SL_BY;
    if (idle) s.lanes = (int)((E + slots - 1) / slots);
  }
  return s;
}

}  // namespace hmc
