"""The word that tells the host which pair kernels have work (csrc/unit_work.cuh),
on the CPU: an answer never belongs to another layout than the one asked for."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
SRC = r"""
#include <atomic>
#include <initializer_list>
#include <thread>
#include "unit_work.cuh"
using namespace abx;
// what a layout of this number holds: all three kinds of layouts in turn
static bool full_of(uint32_t s) { return s % 3 != 0; }
static bool singles_of(uint32_t s) { return s % 3 != 1; }
int main() {
  uint64_t word = 0;
  if (!unit_work(&word, 1).full || !unit_work(&word, 1).singles) return 1;  // nothing written yet
  for (uint32_t s : {1u, 2u, 3u, 0xffffffffu}) {
    word = unit_work_word(s, full_of(s), singles_of(s));
    const UnitWork same = unit_work(&word, s), next = unit_work(&word, s + 1);
    if (same.full != full_of(s) || same.singles != singles_of(s)) return 2;
    if (!next.full || !next.singles) return 3;  // not listed yet: both kernels
  }
  // a writer that is any number of layouts behind the reader, or level with it
  constexpr uint32_t LAST = 300000;
  std::atomic<uint32_t> asked{1};
  std::thread writer([&] {
    for (uint32_t s = 1; s <= LAST; ++s) {
      while (asked.load(std::memory_order_relaxed) < s) {}
      *(volatile uint64_t *)&word = unit_work_word(s, full_of(s), singles_of(s));
    }
  });
  int bad = 0;
  for (uint32_t s = 1; s <= LAST; ++s) {
    asked.store(s, std::memory_order_relaxed);
    for (int k = 0; k < 3; ++k) {
      const UnitWork w = unit_work(&word, s);
      bad += (full_of(s) && !w.full) || (singles_of(s) && !w.singles);
    }
  }
  writer.join();
  return bad ? 4 : 0;
}
"""


def test_work_belongs_to_its_layout(tmp_path):
    src = tmp_path / "unit_work_host.cpp"
    src.write_text(SRC)
    exe = tmp_path / "unit_work_host"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", str(ROOT / "aboria_gb300" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=120).returncode == 0
