// One T per device, made on first use and kept with its owner (a thread's
// streams and events: a stream takes the launches of its own device only, and
// a thread may fit on one device after another).  Plain C++, no CUDA calls.
#pragma once

#include <map>

namespace ct {

template <typename T>
class PerDevice {
 public:
  T& on(int device) { return of_[device]; }

 private:
  std::map<int, T> of_;  // its elements never move
};

}  // namespace ct
