// The position of a ghost from its owner, for the kernels that refresh ghosts.
#pragma once
#include "internal.h"

namespace cacg {

__device__ __forceinline__ int swap_of(const SwapChain &c, int g) {
  int w = 0;
  for (int k = 1; k < c.n; k++)
    if (g >= c.first[k]) w = k;
  return w;
}

// Ghost g's chain of sources back to the owned item (ghost g was sent from
// send[g - nlocal], an owned item or an earlier swap's ghost): the swaps, last
// first, in chain[0..depth), and the owned item as the result.
__device__ __forceinline__ int ghost_chain(const SwapChain &c, const int *__restrict__ send, int nlocal,
                                           int g, int (&chain)[MAX_SWAPS], int &depth) {
  int src = g;
  depth = 0;
  while (src >= nlocal && depth < MAX_SWAPS) {
    chain[depth++] = swap_of(c, src);
    src = send[src - nlocal];
  }
  return src;
}

// ghost g's position: the owner's, the swaps' shifts added in the order the
// swaps ran, the same sum of the same doubles as swap-by-swap communication
__device__ __forceinline__ double4 ghost_position(const double4 *__restrict__ x, const SwapChain &c,
                                                  const int *__restrict__ send, int nlocal, int g) {
  int chain[MAX_SWAPS], depth;
  double4 p = x[ghost_chain(c, send, nlocal, g, chain, depth)];
  for (int k = depth - 1; k >= 0; k--) {
    const int w = chain[k];
    p.x = __dadd_rn(p.x, c.d[w][0]);
    p.y = __dadd_rn(p.y, c.d[w][1]);
    p.z = __dadd_rn(p.z, c.d[w][2]);
  }
  return p;
}

}  // namespace cacg
