// A value that is asked for once and kept, but for failures.
#pragma once

#include <atomic>

namespace tf {

// The value in `slot` (0: not asked yet, else value + 1), or what `ask` returns. A failure (negative) gives 0 and is not kept: the next call
// asks again.
template <class Ask>
int ask_once(std::atomic<int>& slot, Ask ask) {
  const int kept = slot.load(std::memory_order_relaxed);
  if (kept > 0) return kept - 1;
  const int value = ask();
  if (value < 0) return 0;
  slot.store(value + 1, std::memory_order_relaxed);
  return value;
}

}  // namespace tf
