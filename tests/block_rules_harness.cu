// Host program of tests/test_cpu_block_rules.py: for every line "nx ny nz" of its
// input, the planes per block of the node and of the cell pass and the output
// slices per block of the denoiser's convolutions.
#include <cstdio>

#include "k_fields.cuh"
#include "k_denoise.cuh"

int main() {
   rh::GridInfo g = {};
   rh::DnGrid d = {};
   while (std::scanf("%d %d %d", &g.nx, &g.ny, &g.nz) == 3) {
      d.nx = g.nx; d.ny = g.ny; d.nz = g.nz;
      std::printf("%d %d %d\n", rh::layerPlanes(g, rh::ND_Y), rh::layerPlanes(g, rh::NT_Y), rh::tcSlices(d));
   }
}
