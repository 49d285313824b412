// Attributes of kernels (limits and preferences of shared memory).  The runtime
// keeps them per device, so a context keeps its own record of what it has set:
// a record of the process would leave every device but the first without them.
#pragma once

#include <vector>

namespace tms_int
{
  struct KernelAttrs
  {
    struct Entry
    {
      const void* kernel;
      int attr, value;
    };
    std::vector<Entry> done; // some tens of kernels at most: searched in order

    // calls set() unless this record has the value already; set() returns 0 if it worked
    template <class Set>
    auto once(const void* kernel, int attr, int value, const Set& set) -> decltype(set())
    {
      Entry* e = nullptr;
      for (Entry& d : done)
        if (d.kernel == kernel && d.attr == attr) e = &d;
      if (e && e->value == value) return decltype(set())();
      const auto st = set();
      if (st != decltype(set())()) return st;
      if (e) e->value = value;
      else done.push_back(Entry{kernel, attr, value});
      return st;
    }
  };
}
