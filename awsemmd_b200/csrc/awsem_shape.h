// Default launch shape of the fragment-memory kernel (host code).
#pragma once

#include <algorithm>

namespace awsem {

struct FMShape {
  int dsplit;  // work units a residue group: its nd separations in as many chunks
  int grid;    // blocks that take the units; 0: as many as the units fill
};

// Units for `groups` residue groups of `nd` separations each on `sms`
// multiprocessors.
//
// FP64: a separation a unit (units end closer together, and a block can share
// a row) until there are 96 units a multiprocessor, then fewer.  A table
// reaches as far as its longest memory or, on a serving handle, its gamma
// file, so most of many separations hold nothing, and empty units only cost
// their hand-out.  57 separations, six of them filled, us a step by a
// separation a unit / by this rule: 16,000 residues 157 / 147, 32,000 260 /
// 230, 65,000 487 / 382, 131,000 961 / 760.  Six separations: the same up to
// 75,000 residues; 131,000 729 / 719.
//
// FP32: enough units to fill the multiprocessors, two a group at least (1,024
// chains 881 -> 860 us a step), taken by two blocks a multiprocessor up to
// 65,536 residues (two / three: 16,000 89 / 93, 32,000 135 / 139, 43,000 167 /
// 173), by three above (87,000 292 / 288, 131,000 423 / 411, 261,000 835 /
// 785): HBM is saturated then and the pair passes beside it find room (a warp
// a unit there: 300, 432, 836).
inline FMShape fm_shape(bool fp64, int groups, int nd, int sms)
{
  nd = std::max(nd, 1);
  const int g = std::max(groups, 1);
  auto chunks = [&](int units) { return std::min(nd, (units + g - 1) / g); };
  if (fp64) return {chunks(96 * sms), 0};
  return {std::max(std::min(2, nd), chunks(16 * sms)), (g <= 2048 ? 2 : 3) * sms};
}

}  // namespace awsem
