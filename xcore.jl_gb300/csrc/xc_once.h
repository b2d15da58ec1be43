// State that belongs to one CUDA context: what is set, allocated or looked up
// once must be so again on another device, and after a cudaDeviceReset.  Keys are
// xc_context_id() values (xc_internal.cuh), which are never used twice.
#pragma once

#include <map>
#include <mutex>

namespace xc {

// One T per key.  get() returns the key's value, made by make(T*) on first use;
// make returns 0, or an error code, which get() passes on and does not remember.
template <typename T>
class PerKey {
 public:
  template <typename F>
  int get(unsigned long long key, T** out, F&& make) {
    std::lock_guard<std::mutex> lock(mu_);
    auto it = items_.find(key);
    if (it == items_.end()) {
      it = items_.emplace(key, T()).first;
      if (const int st = make(&it->second)) {
        items_.erase(it);
        return st;
      }
    }
    *out = &it->second;                  // (a node's address does not change)
    return 0;
  }

 private:
  std::mutex mu_;
  std::map<unsigned long long, T> items_;
};

}  // namespace xc
