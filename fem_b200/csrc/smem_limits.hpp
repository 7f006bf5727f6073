// smem_limits.hpp -- which kernels' shared memory limits a handle has raised.
//
// The limit belongs to a function on a device: a handle works on one device and
// in one thread at a time, so what it has raised is kept in the handle.  A flag
// per process would leave the limits of a second device as they are, and two
// threads would write it at once.  Handles that share a device raise a function
// to the same size, so their order does not matter.
#pragma once
#include <set>

struct SmemLimits {
  // set(): raises fn's limit, throws if it cannot (it is then tried again).
  template <typename F>
  void raise(const void* fn, F&& set) {
    if (done_.count(fn)) return;
    set();
    done_.insert(fn);
  }

 private:
  std::set<const void*> done_;
};
