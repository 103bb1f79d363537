// Prints, for each domain given as "dim elem tiled smagorinsky partly_solid
// forcing row_nodes planes q", the steps per sweep that sweep.h chooses.
#include <cstdio>

#include "../lbm-c_b200/csrc/sweep.h"

int main() {
  int dim, elem, tiled, smag, partial, force, row, planes, q;
  while (scanf("%d %d %d %d %d %d %d %d %d", &dim, &elem, &tiled, &smag, &partial, &force, &row, &planes, &q) == 9)
    printf("%d\n", lbmc::plan_sweep(planes, (long long)row * q * elem, elem,
                                    lbmc::sweep_plane_limit(dim, elem, tiled, smag, partial, force))
                        .depth);
  return 0;
}
