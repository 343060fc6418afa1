// Shape of a large replica's cell grid, from its bounding box: device code,
// and host code for its test.
#pragma once

#ifdef __CUDACC__
#define AWSEM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define AWSEM_HD inline
#endif

namespace awsem {
namespace dev {

// Cells along each axis, at least `cell` wide (widened until the grid has at
// most `cap` cells, at least one).  For every box, also one that a residue far
// out or at no finite position has made huge: the cells are counted in FP64
// and the widening goes on until they fit (a cell of infinite width at the
// latest), so that nx ny nz is the product as computed here.  Counted in 32
// bits, such a box gave a product that had wrapped, and residues outside the
// cell arrays.
AWSEM_HD void grid_shape(const float lo[3], const float hi[3], int cap, float &cell, int n[3])
{
  while (true) {
    double w[3], tot = 1.0;
    for (int k = 0; k < 3; k++) {
      w[k] = floor((double) ((hi[k] - lo[k]) / cell)) + 1.0;
      if (!(w[k] >= 1.0)) w[k] = 1.0;  // an empty box, or infinite cells
      tot *= w[k];
    }
    if (tot <= cap) {
      for (int k = 0; k < 3; k++) n[k] = (int) w[k];
      return;
    }
    cell *= 1.26f;
  }
}

// the cell of a coordinate along one axis: the nearest one for what lies outside
AWSEM_HD int grid_coord(float p, float o, float inv, int n)
{
  const float c = (p - o) * inv;
  return c >= (float) (n - 1) ? n - 1 : c > 0.f ? (int) c : 0;
}

}  // namespace dev
}  // namespace awsem
