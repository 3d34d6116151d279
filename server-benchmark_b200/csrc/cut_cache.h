// The cuts that a thread used last: a search takes a few microseconds of the host.
#pragma once

namespace awq {

// A call that is cut.  `form`: what is asked of one call, from 0 (with or without scratch, clusters): a call looks up more
// than one form, which lie in slots of their own, so that they do not drive each other out.
struct CutKey {
  int M, slabs, KT, most, device, group, form;
  bool operator==(const CutKey& o) const {
    return M == o.M && slabs == o.slabs && KT == o.KT && most == o.most && device == o.device && group == o.group &&
           form == o.form;
  }
};

template <typename Cut>
class CutCache {
  static constexpr unsigned kSlots = 64;
  struct Entry {
    CutKey key;  // zero-initialised: M 0 is no call
    Cut cut;
  };
  Entry seen[kSlots];

 public:
  template <typename Search>
  Cut get(const CutKey& key, Search search) {
    const unsigned hash = (unsigned)key.M * 2654435761u ^ (unsigned)key.slabs * 40503u ^ (unsigned)key.KT * 97u;
    Entry& e = seen[((hash >> 8) + (unsigned)key.form) % kSlots];
    if (!(e.key == key)) e = Entry{key, search()};
    return e.cut;
  }
};

}  // namespace awq
