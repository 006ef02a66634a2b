"""The table of shared device constants (const_table.h) on the host: plans take no
place of the unplanned calls', what unplanned calls found once they find again, the
plans' part is bounded and gives up the least recently used entry, and an entry is
dropped exactly once, when neither the table nor a plan holds it."""
import shutil
import subprocess

import pytest

from ducc_b200 import build

CXX = shutil.which("g++")
SRC = r"""
#include "const_table.h"
#include <cstdio>
#include <set>
#include <thread>
#include <vector>
using namespace dnufft;
struct V { int k; };
using T = ConstTable<int, V>;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  T t;
  int made = 0;
  std::multiset<int> dropped;
  auto mk = [&](int k) { return [&made, k] { ++made; return new V{k}; }; };
  auto drop = [&](V &v) { dropped.insert(v.k); };
  // many plans, all destroyed again
  for (int k = 0; k < 400; ++k) {
    T::Ptr p = t.for_plan(k, 0, mk(k), drop);
    CHECK(p->k == k);
    t.release(p, drop);
    CHECK(!p);
  }
  CHECK(made == 400 && dropped.size() == 400 - T::RECENT);
  // new geometries of unplanned calls are kept all the same, for good
  const V *first = nullptr;
  for (int r = 0; r < 3; ++r)
    for (int k = 1000; k < 1000 + int(T::KEPT); ++k) {
      const V *v = t.for_call(k, 0, mk(k));
      CHECK(v && v->k == k);
      if (k == 1000) { CHECK(!first || v == first); first = v; }
      for (int j = 0; j < 150; ++j) {
        T::Ptr p = t.for_plan(2000 + (r * 70 + j), 0, mk(2000), drop);
        t.release(p, drop);
      }
    }
  CHECK(t.for_call(1, 0, mk(1)) == nullptr);
  CHECK(t.for_call(1000, 0, mk(1000)) == first);
  for (int k = 1000; k < 1000 + int(T::KEPT); ++k) CHECK(dropped.count(k) == 0);
  // a plan shares the calls' entry, and its release does not drop it
  int before = made;
  T::Ptr s = t.for_plan(1000, 0, mk(1000), drop);
  CHECK(s.get() == first && made == before);
  t.release(s, drop);
  CHECK(dropped.count(1000) == 0);
  // least recently used first; held entries survive their eviction, then are dropped once
  T u;
  dropped.clear();
  T::Ptr a = u.for_plan(0, 0, mk(0), drop), b = u.for_plan(0, 0, mk(0), drop);
  CHECK(a == b);
  for (int k = 1; k < int(T::RECENT); ++k) { T::Ptr p = u.for_plan(k, 0, mk(k), drop); u.release(p, drop); }
  CHECK(dropped.empty());
  before = made;
  { T::Ptr p = u.for_plan(1, 0, mk(1), drop); u.release(p, drop); }   // 1 is young again
  CHECK(made == before);
  { T::Ptr p = u.for_plan(10000, 0, mk(10000), drop); u.release(p, drop); }   // evicts 0 (held)
  { T::Ptr p = u.for_plan(10001, 0, mk(10001), drop); u.release(p, drop); }   // evicts 2
  CHECK(dropped == std::multiset<int>{2});
  u.release(a, drop);
  CHECK(dropped.count(0) == 0);
  u.release(b, drop);
  CHECK(dropped.count(0) == 1);
  // an unplanned call takes over an entry that plans made
  before = made;
  CHECK(u.for_call(1, 0, mk(1))->k == 1 && made == before);
  // devices apart
  { T::Ptr p = u.for_plan(10001, 1, mk(10001), drop); CHECK(made == before + 1); u.release(p, drop); }
  // from several threads
  std::vector<std::thread> th;
  std::mutex m;
  int bad = 0;
  for (int i = 0; i < 8; ++i)
    th.emplace_back([&, i] {
      for (int r = 0; r < 2000; ++r) {
        const int k = (r * 13 + i) % 300;
        T::Ptr p = u.for_plan(k, 0, [k] { return new V{k}; }, [&](V &v) { v.k = -1; });
        if (p->k != k) { std::lock_guard<std::mutex> l(m); ++bad; }
        u.release(p, [&](V &v) { v.k = -1; });
      }
    });
  for (auto &x : th) x.join();
  CHECK(bad == 0);
  std::puts("ok");
  return 0;
}
"""


@pytest.mark.skipif(CXX is None, reason="needs g++")
def test_shared_constants(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([CXX, "-std=c++17", "-O1", "-pthread", "-I" + build.CSRC, "-o", str(exe),
                    str(src)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
