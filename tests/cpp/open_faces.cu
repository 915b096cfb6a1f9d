// dilateTile's device check on one brick at a boundary that remaps cells: prints
// the error word for every boundary kind, face and neighbour (allocated or not)
// with one defined cell on that face.  Input and output of a line:
// kind face allocated error.
#include <cstdio>

#include "vlsg_frontier.cuh"

using namespace vlsg;

__global__ void dilate(Topo t, const uint64_t *mask, int face, int neighbour) {
  int nb[6] = {0, 0, 0, 0, 0, 0};
  nb[face] = neighbour;
  const int z = threadIdx.x & 7;
  const bool on = threadIdx.x < 8;
  dilateTile<true>(t, mask, 0, nb, z, on ? mask[z] : 0ull, on, true);
}

int main() {
  uint64_t *mask;
  int *err, *slotBrick;
  if (cudaMallocManaged(&mask, 8 * sizeof(uint64_t)) || cudaMallocManaged(&err, sizeof(int)) ||
      cudaMallocManaged(&slotBrick, sizeof(int)))
    return 1;
  slotBrick[0] = 0;
  for (int bc = 0; bc <= 4; ++bc)
    for (int face = 0; face < 6; ++face)
      for (int allocated = 0; allocated < 2; ++allocated) {
        GridDev g{};
        const int d = face / 2;
        const bool upper = face & 1;
        for (int k = 0; k < 3; ++k) {
          // a brick of 8 cells at 0 in a grid from 0 to 6 (all of it within the
          // brick) in the direction of the boundary, far wider in the others
          g.org[k] = 0, g.nb[k] = 1;
          g.bc[k] = k == d ? bc : VLSG_INFINITE_BOUNDARY;
          g.gmin[k] = k == d ? 0 : -64;
          g.gmax[k] = k == d ? 6 : 64;
        }
        const int last = bc == VLSG_PERIODIC_BOUNDARY ? 5
                         : bc == VLSG_REFLECTIVE_BOUNDARY || bc == VLSG_NEG_INFINITE_BOUNDARY ? 6 : 7;
        int c[3] = {3, 3, 3};
        c[d] = upper ? last : 0;
        for (int z = 0; z < 8; ++z) mask[z] = 0ull;
        mask[c[2]] = 1ull << (c[1] * 8 + c[0]);
        *err = 0;
        Topo t{g, nullptr, slotBrick, nullptr, nullptr, nullptr, nullptr, err};
        dilate<<<1, 32>>>(t, mask, face, allocated ? 0 : -1);
        if (cudaDeviceSynchronize() != cudaSuccess) return 1;
        std::printf("%d %d %d %d\n", bc, face, allocated, *err);
      }
  return 0;
}
