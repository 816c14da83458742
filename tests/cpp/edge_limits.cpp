// The largest meshes of the FP64 path: n_edges padded, or -1 where it is refused.
#include <stdexcept>

#include "slot_planes.hpp"

extern "C" long long padded(int n_edges) {
  try {
    return splash::padded_edges(n_edges);
  } catch (const std::runtime_error&) {
    return -1;
  }
}
extern "C" long long max_adjoint_sides() { return (long long)splash::kMaxAdjointSides; }
