// Which of the two pair kernels of a layout have work (pairs.cu), as one 64-bit
// word in mapped host memory: the device writes it with one store once the units
// are listed, the host reads it with one load before a launch.  A load sees a whole
// word, so the answer always belongs to the layout number beside it, in whatever
// order the processor and the compiler leave other accesses (a number and counts
// as separate words need release and acquire ordering on both sides).
#pragma once

#include <stdint.h>

namespace abx {

constexpr uint64_t UNIT_WORK_FULL = 1, UNIT_WORK_SINGLES = 2;

// seq: the layout's number, from 1 on (0: nothing written yet)
constexpr uint64_t unit_work_word(uint32_t seq, bool full, bool singles) {
  return (uint64_t)seq << 32 | (full ? UNIT_WORK_FULL : 0) | (singles ? UNIT_WORK_SINGLES : 0);
}

struct UnitWork {
  bool full, singles;  // true where the kernel has, or may have, work
};

inline UnitWork unit_work(const uint64_t *word, uint32_t seq) {
  const uint64_t w = __atomic_load_n(word, __ATOMIC_RELAXED);
  const bool known = (uint32_t)(w >> 32) == seq;
  return {!known || (w & UNIT_WORK_FULL) != 0, !known || (w & UNIT_WORK_SINGLES) != 0};
}

}  // namespace abx
