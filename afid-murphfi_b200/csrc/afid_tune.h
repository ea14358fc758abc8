// afid_tune.h — where the K1 autotuner's launches keep their four RK3 histories (host only).
#pragma once
#include <cstddef>

namespace afid {

struct TunePlace {
  int mem;        // 0, 1: the buffers that are dead between substeps; 2: scratch
  size_t offset;  // bytes
};

// Four disjoint places of `bytes` each, in the dead buffers (dead[0], dead[1] bytes) as far as they hold
// them.  Returns the scratch bytes that the others need.
inline size_t tune_places(size_t bytes, const size_t (&dead)[2], TunePlace (&place)[4]) {
  size_t used[3] = {0, 0, 0};
  for (TunePlace &p : place) {
    p.mem = used[0] + bytes <= dead[0] ? 0 : used[1] + bytes <= dead[1] ? 1 : 2;
    p.offset = used[p.mem];
    used[p.mem] += bytes;
  }
  return used[2];
}

}  // namespace afid
