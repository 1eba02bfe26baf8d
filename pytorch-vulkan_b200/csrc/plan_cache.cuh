// Plans kept per thread: a layer's plan depends on its geometry alone, and a network calls the same layers again and again.  One convolution
// call consults a dozen plans (is the kernel applicable, how much workspace, which tiles); made anew each time they took 10 to 60 us of
// host time, as long as a small layer takes on the device.
#pragma once
#include <cstring>
#include <memory>

#include "common.cuh"

namespace b200 {

// A table of a fixed size, four places to a hash value: what falls on four others' places replaces one of them in turn.  One object per thread
// (thread_local); the entries are allocated with the first plan.  A network of fifty convolutions asks for a hundred plans a training step (forward
// and dInput are two): of 104 lookups for ResNet-50 at batch 32, 32 places of one entry each missed 34 in every step, 128 places of four none.
template <typename Plan>
class PlanCache {
  static constexpr unsigned SETS = 128, WAYS = 4;
  struct Entry {
    ConvGeom g;
    size_t extra;   // whatever else the plan depends on
    int sms = 0;    // SMs of the device the plan was made for; 0: empty
    Plan plan;
  };
  std::unique_ptr<Entry[]> entries_;
  unsigned next_ = 0;

 public:
  template <typename Make>
  const Plan& get(const ConvGeom& g, size_t extra, Make&& make) {
    static_assert(sizeof(ConvGeom) % sizeof(unsigned) == 0, "hashed and compared as words without padding");
    unsigned words[sizeof(ConvGeom) / sizeof(unsigned)], hash = (unsigned)extra * 2654435761u;
    memcpy(words, &g, sizeof words);
    for (unsigned w : words) hash = (hash ^ w) * 16777619u;
    if (!entries_) entries_.reset(new Entry[SETS * WAYS]);
    Entry* set = &entries_[(hash ^ hash >> 15) % SETS * WAYS];
    const int sms = sm_count();
    Entry* place = nullptr;
    for (unsigned i = 0; i < WAYS; ++i) {
      Entry& e = set[i];
      if (e.sms == sms && e.extra == extra && memcmp(&e.g, &g, sizeof g) == 0) return e.plan;
      if (e.sms == 0 && !place) place = &e;
    }
    if (!place) place = &set[next_++ % WAYS];
    place->sms = 0;
    place->plan = make();
    place->g = g; place->extra = extra; place->sms = sms;
    return place->plan;
  }
};

}  // namespace b200
