"""The host block a topology is laid out in (csrc/pinned_arena.h), against a fake of pinned memory.

It takes pageable memory where pinned memory is refused, asks for the exact size where twice the old
one is refused, grows geometrically, and gives every block back once, to where it came from.
"""
from __future__ import annotations

import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cassert>
#include <cstring>
#include "pinned_arena.h"

struct Fake {
  static size_t limit;         // larger requests are refused
  static int made, freed, asked;
  static void* allocate(size_t n) {
    ++asked;
    if (n > limit) return nullptr;
    ++made;
    return std::malloc(n);
  }
  static void release(void* p) {
    ++freed;
    std::free(p);
  }
};
size_t Fake::limit = 0;
int Fake::made = 0, Fake::freed = 0, Fake::asked = 0;

template <class A> void fill(A& a, size_t n) {
  char* p = a.template take<char>(n);
  std::memset(p, 7, n);
}

int main() {
  {
    xtb::HostArena<Fake> a;    // refused: pageable, and usable
    assert(a.reset(1000) && !a.pinned() && a.capacity() == 1000);
    fill(a, 1000);
    Fake::limit = 3000;        // pinned memory again: twice the size
    assert(a.reset(1200) && a.pinned() && a.capacity() == 2000);
    fill(a, 1200);
    assert(a.reset(2900) && a.pinned() && a.capacity() == 2900);   // 4000 refused, 2900 not
    fill(a, 2900);
    assert(a.reset(5000) && !a.pinned() && a.capacity() == 5000);
    fill(a, 5000);
  }
  assert(Fake::made == 2 && Fake::freed == 2);
  Fake::limit = size_t(1) << 40;
  Fake::asked = Fake::made = Fake::freed = 0;
  {
    xtb::HostArena<Fake> a;    // a thousand growing topologies: a dozen blocks
    for (size_t n = 64; n <= 64000; n += 64) {
      assert(a.reset(n));
      fill(a, n);
    }
    assert(a.capacity() < 2 * 64000);
    assert(a.reset(10) && a.capacity() >= 64000);   // and is kept
  }
  assert(Fake::asked == Fake::made && Fake::made <= 12 && Fake::freed == Fake::made);
  xtb::HostArena<Fake> a;
  assert(a.reset(3 * 64));
  char* first = a.take<char>(1);
  int* second = a.take<int>(3);
  assert(reinterpret_cast<char*>(second) == first + 64 && a.take<char>(64) == first + 128);
  return 0;
}
"""


def test_arena(tmp_path):
    source = tmp_path / "arena.cpp"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-fsanitize=address,undefined",
                    "-I", str(ROOT / "xtbloom_b200" / "csrc"), str(source), "-o", str(tmp_path / "arena")], check=True)
    subprocess.run([str(tmp_path / "arena")], check=True)
