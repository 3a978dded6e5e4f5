// Whether a step's kernel made its step, for the launch that finishes it.
#pragma once

#ifdef __CUDACC__
#define APO_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define APO_HOST_DEVICE inline
#endif

namespace apo {

// The kinetic energy, the averages and the counters of a step are formed by a
// launch of their own beside the next step's forces.  Those forces can set the
// list's error word, so that launch must not ask the word whether the step
// was made: the state would have moved by a step that the counters leave
// out.  The step's own kernel, which no forces run beside, decides and says
// so here; the finishing launch takes the record, so a step that was not made
// is finished by nobody and one that was by exactly one launch.
struct StepRecord {
  unsigned made;
};

APO_HOST_DEVICE void record_step(StepRecord &r) { r.made = 1u; }

APO_HOST_DEVICE bool take_step(StepRecord &r) {
  const bool made = r.made != 0u;
  r.made = 0u;
  return made;
}

}  // namespace apo
