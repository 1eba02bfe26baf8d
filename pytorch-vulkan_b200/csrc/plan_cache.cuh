// Plans kept per thread: a layer's plan depends on its geometry alone, and a network calls the same layers again and again.  One convolution
// call consults a dozen plans (is the kernel applicable, how much workspace, which tiles); made anew each time they took 10 to 60 us of
// host time, as long as a small layer takes on the device.
#pragma once
#include <cstring>

#include "common.cuh"

namespace b200 {

// A direct-mapped table of a fixed size: a geometry that falls on another's place replaces it.  One object per thread (thread_local).
template <typename Plan>
class PlanCache {
  static constexpr unsigned SIZE = 32;
  struct Entry {
    ConvGeom g;
    size_t extra;   // whatever else the plan depends on
    int sms = 0;    // SMs of the device the plan was made for; 0: empty
    Plan plan;
  };
  Entry entries_[SIZE];

 public:
  template <typename Make>
  const Plan& get(const ConvGeom& g, size_t extra, Make&& make) {
    static_assert(sizeof(ConvGeom) % sizeof(unsigned) == 0, "hashed and compared as words without padding");
    unsigned words[sizeof(ConvGeom) / sizeof(unsigned)], hash = (unsigned)extra * 2654435761u;
    memcpy(words, &g, sizeof words);
    for (unsigned w : words) hash = (hash ^ w) * 16777619u;
    Entry& e = entries_[(hash ^ hash >> 15) % SIZE];
    const int sms = sm_count();
    if (e.sms != sms || e.extra != extra || memcmp(&e.g, &g, sizeof g) != 0) {
      e.sms = 0;
      e.plan = make();
      e.g = g; e.extra = extra; e.sms = sms;
    }
    return e.plan;
  }
};

}  // namespace b200
