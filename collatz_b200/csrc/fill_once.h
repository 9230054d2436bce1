// fill_once.h -- device tables that every context of a device shares are written once.
#pragma once
#include <mutex>

namespace cz {

// Runs fill and then mark unless ready says that both have run before; ready(bool*), fill() and mark()
// return 0 or an error, which ends the call with nothing marked.  What they start on the device must
// have ended when they return: kernels of contexts made earlier read the tables without any order
// with this one, so that nothing may be written once another context has seen them ready.  The mark
// belongs beside the tables, on the device: a device that is reset loses both.
template <class Ready, class Fill, class Mark>
auto fill_once(Ready ready, Fill fill, Mark mark) -> decltype(fill()) {
  static std::mutex m;
  std::lock_guard<std::mutex> g(m);
  bool done = false;
  auto e = ready(&done);
  if (e || done) return e;
  e = fill();
  return e ? e : mark();
}

}  // namespace cz
