// Largest thread-block cluster that a kernel can be launched with.
#pragma once

namespace b200pa {

// `places(n)`: how many clusters of n CTAs the GPU has room for at once; 0 or an error code below it where
// it has none.  Clusters of 16 are not portable: a GPU with fewer SMs in its GPCs (partitioned, or another
// part) takes smaller ones.
template <typename F>
int largest_cluster(F&& places) {
  for (int n = 16; n > 1; n /= 2)
    if (places(n) > 0) return n;
  return 1;
}

}  // namespace b200pa
