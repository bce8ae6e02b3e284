// One device buffer per device ordinal, grown on demand and kept for the life of
// the process.  The runtime calls come from Api (current device, allocation,
// release), so that the bookkeeping can be tested without a GPU.  Not
// synchronised: the owner's lock covers a call and the buffer's use.
#pragma once
#include <cstddef>
#include <map>

namespace xtg {

template <class Api>
class PerDevice {
 public:
  // the current device's buffer of at least `need` bytes; *fresh: just allocated
  // (a larger one replaces a smaller one, whose contents are lost)
  typename Api::Error get(size_t need, void **out, bool *fresh = nullptr) {
    int dev = 0;
    if (fresh) *fresh = false;
    typename Api::Error e = Api::device(&dev);
    if (e != Api::ok) return e;
    Slot &s = slots_[dev];
    if (need > s.bytes) {
      if (s.p) Api::release(s.p);
      s = Slot{};
      if ((e = Api::allocate(&s.p, need)) != Api::ok) {
        s = Slot{};
        return e;
      }
      s.bytes = need;
      if (fresh) *fresh = true;
    }
    *out = s.p;
    return Api::ok;
  }

 private:
  struct Slot {
    void *p = nullptr;
    size_t bytes = 0;
  };
  std::map<int, Slot> slots_;
};

}  // namespace xtg
