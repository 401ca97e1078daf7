// Device scratch that only makes a call faster.
#pragma once
#include <c10/util/Exception.h>
#include <torch/types.h>

namespace ody {

// `want` bytes on `like`'s device from the caching allocator, or none when there is no memory left for them: a call that fits
// without its scratch still runs, unsplit.
struct OptionalScratch {
  at::Tensor t;
  int64_t bytes = 0;
  OptionalScratch(int64_t want, const at::Tensor& like) {
    if (want <= 0) return;
    try {
      t = at::empty({want}, like.options().dtype(at::kByte));
      bytes = want;
    } catch (const c10::OutOfMemoryError&) {
    }
  }
  void* ptr() const { return bytes > 0 ? t.data_ptr() : nullptr; }
};

}  // namespace ody
