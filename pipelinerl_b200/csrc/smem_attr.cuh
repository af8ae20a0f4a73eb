// The largest dynamic shared memory that a kernel may be launched with is an attribute of the function on each device, and setting it
// to less takes the larger size back.  One static SmemAttr per launch site remembers what is granted.  Host code only, no CUDA in it:
// the setter comes from the caller.
#pragma once
#include <mutex>

namespace prl {

constexpr int kMaxDevices = 16;
struct SmemAttr {
  std::mutex lock;
  int bytes[kMaxDevices];
};

// At least `smem` bytes on device `dev`: `set(smem)` returns 0 or an error, which is handed on.  Comparing, setting and noting are one
// step: a launch site whose size depends on the call (the products' ring on the k-blocks, the decode attention's buffers on the batch) is
// reached by several threads at once, and a smaller size that was set last under a larger one that was noted failed every larger launch.
template <typename Set>
inline auto raise_smem(SmemAttr& st, int dev, int smem, Set set) -> decltype(set(smem)) {
  std::lock_guard<std::mutex> hold(st.lock);
  if (st.bytes[dev] >= smem) return {};
  const auto e = set(smem);
  if (e == decltype(e){}) st.bytes[dev] = smem;
  return e;
}

}  // namespace prl
