"""The order among calls that share one of the library's buffers (csrc/use_order.h), with streams and events
that only record what they are asked."""
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]

FAKE = r'''
#include "use_order.h"
#include <cstdio>
#include <string>
using namespace ssb;
// stream 2 is one handle of several streams; generation: stream handles 5 and up come back as other streams
static int generation = 0;
// every call leaves a letter and the stream's (or the event's) number in `said`
static std::string said;
static int fail_record = 0, fail_create = 0, events = 0;
struct Fake {
  using Stream = int;
  using Event = int;
  using Error = int;
  static int create(int& e) {
    if (fail_create) return 2;
    e = ++events;
    return 0;
  }
  static int wait(int s, int e) { said += "w" + std::to_string(s) + "/" + std::to_string(e) + " "; return 0; }
  static int record(int e, int s) {
    if (fail_record) return 9;
    said += "r" + std::to_string(s) + "/" + std::to_string(e) + " ";
    return 0;
  }
  static int sync(int e) { said += "h" + std::to_string(e) + " "; return 0; }
  static void sync_stream(int s) { said += "s" + std::to_string(s) + " "; }
  static uint64_t id(int s) { return s == 2 ? 0 : s + 100 * generation; }
  static void destroy(int e) { said += "d" + std::to_string(e) + " "; }
};
static bool was(const char* what) {
  const bool same = said == what;
  if (!same) std::printf("said %s, not %s\n", said.c_str(), what);
  said.clear();
  return same;
}
'''


def _run(tmp_path, body, before=""):
    src = tmp_path / "t.cpp"
    src.write_text(FAKE + before + "int main() {\n" + body + '\n  std::puts("ok");\n  return 0;\n}\n')
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(ROOT / "ssblasex_b200" / "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout)


def test_a_call_waits_for_the_one_before(tmp_path):
    """Whatever its stream, unless that is known to be the same: equal handles need not be one stream. An event
    that cannot be recorded is replaced by a wait of the host."""
    _run(tmp_path, r'''
  UseOrder<Fake> o;
  if (o.begin(5) || !was("")) return 1;              // nothing before it
  o.end(5);
  if (!was("r5/1 ") || o.begin(5) || !was("")) return 2;   // the same stream is in order by itself
  o.end(5);
  if (!was("r5/1 ") || o.begin(7) || !was("w7/1 ")) return 3;
  o.end(7);
  generation = 1;
  if (!was("r7/1 ") || o.begin(7) || !was("w7/1 ")) return 4;   // the same handle, another stream
  o.end(7);
  o.begin(2);
  o.end(2);
  if (!was("r7/1 w2/1 r2/1 ") || o.begin(2) || !was("w2/1 ")) return 5;   // a handle of several streams
  fail_record = 1;
  o.end(2);
  if (!was("s2 ")) return 6;
  fail_record = 0;
  if (o.idle() || !was("h1 ") || o.idle() || !was("")) return 7;
  if (o.begin(5) || !was("")) return 8;              // idle: nothing to wait for
  o.end(5);
  o.destroy();
  if (!was("r5/1 d1 ")) return 9;
  fail_create = 1;
  UseOrder<Fake> p;
  if (p.begin(5) != 2 || p.made) return 10;
''')


def test_a_use_ends_on_every_way_out(tmp_path):
    """A call whose second launch fails has its first queued: the next call, on another stream, waits for it. A
    call whose wait failed queued nothing."""
    _run(tmp_path, r'''
  UseOrder<Fake> o;
  if (call(o, 5, 2) != 7 || !was("l l r5/1 ")) return 1;
  if (call(o, 6, 9) != 0 || !was("w6/1 l l l r6/1 ")) return 2;
  fail_create = 1;
  UseOrder<Fake> p;
  if (call(p, 5, 9) != 2 || !was("") || p.in_use) return 3;
''', before=r'''
// a call of three launches, of which number `bad` is refused
static int call(UseOrder<Fake>& o, int st, int bad) {
  const Use<Fake> use(o, st);
  if (use.error()) return use.error();
  for (int i = 1; i <= 3; ++i) {
    said += "l ";
    if (i == bad) return 7;
  }
  return 0;
}
''')
