"""The growth of the wavefront's state (csrc/vt_grow.h) against a device that holds only so much: what a caller can do without
never costs another one the buffer that it has, and a refusal is not asked for again while there is no more room."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r'''
#include <cassert>
#include <cstdlib>
#include <map>

#include "vt_grow.h"

struct Dev {
  size_t total = 0, used = 0, asked = 0, freed = 0, synced = 0;
  std::map<void*, size_t> held;
  void* alloc(size_t n) {
    asked++;
    if (used + n > total) return nullptr;
    void* p = std::malloc(1);
    held[p] = n;
    used += n;
    return p;
  }
  void free(void* p) {
    assert(held.count(p) && synced > freed);   // only after a wait for the work on it
    used -= held[p];
    held.erase(p);
    std::free(p);
    freed++;
  }
  void sync() { synced++; }
  size_t room() { return total - used; }
};

int main() {
  Dev d;
  d.total = 1000;
  vtapi::GrowBuffer b;
  assert(b.grow(d, 300) && b.cap == 300 && d.used == 300);
  void* const p = b.p;
  // 800 do not fit beside the 300: the 300 stay, and nobody asks again
  for (int frame = 0; frame < 5; frame++) assert(!b.try_grow(d, 800) && b.p == p && b.cap == 300);
  assert(d.asked == 2 && d.freed == 0 && d.synced == 0);
  // less than was refused is tried, more is not
  assert(!b.try_grow(d, 900) && d.asked == 2);
  assert(b.try_grow(d, 600) && b.cap == 600 && d.used == 600 && d.freed == 1);
  // what cannot be done without takes the old one's place
  assert(b.grow(d, 700) && b.cap == 700 && d.used == 700);
  assert(b.grow(d, 200) && b.cap == 700);
  // a refusal holds until there is more room
  assert(!b.try_grow(d, 950));
  size_t asked = d.asked;
  assert(!b.try_grow(d, 950) && d.asked == asked);
  d.total = 2000;
  assert(b.try_grow(d, 950) && b.cap == 950 && d.used == 950);
  // and what is not there at all leaves an empty buffer, never one that is smaller than its cap says
  assert(!b.grow(d, 3000) && b.p == nullptr && b.cap == 0 && d.used == 0);
  assert(b.grow(d, 100) && b.cap == 100);
  return 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ absent")
def test_growth_keeps_what_others_count_on(tmp_path):
    src, exe = tmp_path / "grow.cpp", tmp_path / "grow"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "veridien-twin_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
