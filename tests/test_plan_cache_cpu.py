"""Which plans of grouped calls stay (csrc/plan_cache.h): the most recently used ones within the bounds, and
those that a CUDA graph holds whatever comes after."""
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]
SRC = r'''
#include "plan_cache.h"
#include <cstdio>
#include <set>
using namespace ssb;
static std::set<int> alive;
struct Plan {
  int shapes;
  size_t scratch;
  unsigned long tick = 0;
  bool captured = false;
  Plan(int s, size_t b) : shapes(s), scratch(b) { alive.insert(s); }
  ~Plan() { alive.erase(shapes); }
};
using Cache = PlanCache<Plan, 4, 1000>;
// a call of these shapes, as the library makes it
static Plan* call(Cache& c, int shapes, size_t scratch, bool captured) {
  Plan* p = c.find(captured, [&](const Plan& x) { return x.shapes % 1000 == shapes % 1000; });
  if (!p) {
    auto n = std::make_unique<Plan>(shapes, scratch);
    c.make_room(scratch);
    p = c.add(std::move(n));
  }
  c.use(*p);
  if (captured) p->captured = true;
  return p;
}
int main() {
  Cache c;
  for (int s = 0; s < 6; ++s) call(c, s, 10, false);
  if (alive != std::set<int>{2, 3, 4, 5}) return 1;
  call(c, 2, 10, false);
  call(c, 6, 10, false);                                   // 3 was used longest ago
  if (alive != std::set<int>{2, 4, 5, 6}) return 2;
  call(c, 7, 985, false);                                  // too much beside any two others
  if (alive != std::set<int>{6, 7}) return 3;
  call(c, 8, 5000, false);                                 // above the bound by itself: alone
  if (alive != std::set<int>{8}) return 4;
  Plan* held = call(c, 8, 5000, true);
  if (!held->captured || c.size() != 1) return 5;
  // neither other shapes nor their scratch drop it, and it does not count against them
  for (int s = 10; s < 30; ++s) call(c, s, 400, false);
  if (alive != std::set<int>{8, 28, 29}) return 6;
  // an ordinary call of its shapes has a plan of its own; a call under capture has the graph's
  Plan* own = call(c, 1008, 10, false);
  if (own == held || own->captured || call(c, 2008, 10, true) != held) return 7;
  if (call(c, 1008, 10, false) != own) return 8;
  c.clear();
  if (!alive.empty()) return 9;
  std::puts("ok");
  return 0;
}
'''


def test_plans_kept(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(ROOT / "ssblasex_b200" / "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout)
