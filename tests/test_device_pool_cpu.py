"""The bookkeeping of device memory (csrc/device_pool.cuh) against a fake allocator of 100 bytes."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gradwave_b200" / "csrc"

FAKE = """
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <map>
#include "device_pool.cuh"

struct Fake {
  static inline std::map<void*, size_t> live;
  static inline size_t room = 100;
  static inline int calls = 0;
  static bool alloc(void** p, size_t n) {
    ++calls;
    if (n > room) return false;
    *p = std::malloc(1);
    live[*p] = n;
    room -= n;
    return true;
  }
  static void free(void* p) {
    assert(live.count(p));
    room += live[p];
    live.erase(p);
    std::free(p);
  }
};
using Pool = gwb::DevicePool<Fake>;
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\\n", __LINE__, #x); return 1; }
"""

KEPT = """
int main() {
  Pool pool;
  void *w = nullptr, *p = nullptr, *q = nullptr;
  size_t n = 0, have = 0;
  pool.handles(0, 2);
  CHECK(pool.ensure(0, &w, &have, 60) && Fake::room == 40);
  pool.give(0, w, have);                       // a destroyed handle's scratch stays ...
  CHECK(Fake::room == 40);
  CHECK(!pool.take(0, 61, &n) && !pool.take(1, 1, &n));
  CHECK(pool.alloc(0, &p, 30) && Fake::room == 10);
  CHECK(pool.alloc(0, &q, 50) && Fake::room == 20);   // ... until any allocation needs its room
  CHECK(!pool.take(0, 0, &n));
  void* r = &n;
  CHECK(!pool.alloc(0, &r, 21) && r == nullptr && Fake::room == 20);
  have = 30;
  CHECK(!pool.ensure(0, &p, &have, 60) && p == nullptr && have == 0);
  CHECK(pool.ensure(0, &p, &have, 40) && have == 40);
  pool.give(0, p, 40);
  pool.give(0, q, 50);                         // the larger of two stays
  CHECK(Fake::room == 50 && pool.take(0, 50, &n) == q && n == 50);
  pool.give(0, q, 50);
  pool.handles(0, -1);
  CHECK(Fake::room == 50);
  pool.handles(0, -1);                         // the last handle takes it along
  CHECK(Fake::room == 100 && Fake::live.empty());
  return 0;
}
"""

ALL_OR_NONE = """
int main() {
  Pool pool;
  void *a = nullptr, *b = nullptr, *c = nullptr;
  CHECK(!pool.alloc_all(0, {{&a, 40}, {&b, 40}, {&c, 40}}));
  CHECK(!a && !b && !c && Fake::room == 100 && Fake::live.empty());
  CHECK(pool.alloc_all(0, {{&a, 40}, {&b, 40}, {&c, 20}}) && a && b && c && Fake::room == 0);
  return 0;
}
"""

CHUNKS = """
int main() {
  Pool pool;
  gwb::ChunkScratch w;
  size_t n = 0;
  CHECK(pool.chunk(0, w, 7, 10, 40, 20) == 4 && w.bytes == 40);      // two chunks of 4 and 3
  CHECK(pool.chunk(0, w, 100, 10, 5, 2) == 1 && w.bytes == 40);      // one band at least
  CHECK(pool.chunk(0, w, 30, 10, 300, 20) == 4 && w.bytes == 40);    // no room for 300: what it held
  const int calls = Fake::calls;
  for (int i = 0; i < 3; ++i) CHECK(pool.chunk(0, w, 30, 10, 300, 20) == 4);
  CHECK(Fake::calls == calls);                                       // and no further attempt
  CHECK(pool.chunk(0, w, 6, 10, 300, 20) == 6 && w.bytes == 60);     // a smaller one may be had
  CHECK(pool.chunk(0, w, 30, 10, 300, 20) == 6 && w.bytes == 60);
  gwb::ChunkScratch v;
  CHECK(pool.chunk(0, v, 30, 10, 300, 20) == 2 && v.bytes == 20);    // the low budget
  gwb::ChunkScratch u;
  CHECK(pool.chunk(0, u, 30, 21, 300, 20) == 0 && !u.p && u.bytes == 0);
  Fake::free(v.p);
  Fake::free(w.p);
  w = {};
  Fake::room = 0;                                                    // no allocation at all (a stream capture) ...
  CHECK(pool.chunk(0, w, 9, 10, 90, 20) == 0 && w.bytes == 0);
  Fake::room = 100;
  CHECK(pool.chunk(0, w, 9, 10, 90, 20) == 9 && w.bytes == 90);      // ... says nothing about the room
  Fake::free(w.p);
  w = {};
  CHECK(pool.chunk(0, w, 6, 10, 300, 20) == 6);
  CHECK(pool.chunk(0, u, 30, 21, 300, 20) == 1 && u.bytes == 21);    // asked for again
  pool.handles(0, 1);
  pool.give(0, w.p, w.bytes);
  CHECK(pool.chunk(0, u, 3, 20, 300, 20) == 3 && u.bytes == 60 && Fake::room == 40);   // a kept buffer taken over
  return 0;
}
"""


def _run(tmp_path, main):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text(FAKE + main)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp"), "-pthread"], check=True)
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr


def test_kept_scratch_is_given_back(tmp_path):
    _run(tmp_path, KEPT)


def test_tables_of_a_set_come_all_or_none(tmp_path):
    """gwb_ham_set_overlap tells by its first table whether it has them: a set that a failure left incomplete would
    send the next call to a null one."""
    _run(tmp_path, ALL_OR_NONE)


def test_chunks_when_memory_is_short(tmp_path):
    _run(tmp_path, CHUNKS)


def test_every_allocation_of_a_handle_uses_the_pool():
    """No handle allocates past the pool: cudaMalloc is called in its Api alone."""
    for src in sorted(CSRC.glob("*.cu*")):
        assert src.read_text().count("cudaMalloc(") == (src.name == "ham_apply.cu"), src.name
