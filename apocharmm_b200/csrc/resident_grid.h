// Grid sizes of persistent launches, asked of the device once.
#pragma once

namespace apo {

// Blocks of a persistent launch: all that fit, and as many as leave room on
// every SM for other kernels.
struct ResidentGrid {
  int full = 0, shared = 0;
};

// The answer of `query`, asked once per kernel form (each launch function has
// a lambda, and so an instance, of its own) by the thread that comes first;
// threads that come meanwhile wait for the whole answer.  (Two plain statics,
// one of them doubling as "known", let a second host thread launch with the
// other one still zero.)
template <typename Query>
const ResidentGrid &resident_grid(Query query) {
  static const ResidentGrid g = query();
  return g;
}

}  // namespace apo
