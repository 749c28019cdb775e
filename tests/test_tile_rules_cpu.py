"""The rules that choose a tile (csrc/tile_rules.h), at the measured sides of their lines."""
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]

# m, n, k, batch, beta != 0, narrow tiles were the faster ones (by more than the runs' spread), on 148 SMs
I8 = [
    (2048, 2048, 2048, 1, 0, 0), (2048, 2048, 8192, 1, 1, 0), (1024, 4096, 4096, 1, 0, 0), (1024, 1024, 1024, 4, 0, 0),
    (1024, 2048, 2048, 2, 1, 0), (1536, 2048, 4096, 1, 0, 0), (512, 512, 4096, 12, 0, 0), (2304, 2048, 16384, 1, 0, 0),
    (512, 256, 4096, 1, 0, 1), (1024, 1024, 4096, 1, 0, 1), (2048, 1024, 4096, 1, 0, 1), (512, 512, 8192, 7, 0, 1),
    (512, 256, 16384, 1, 0, 1), (1024, 512, 16384, 1, 0, 1), (1536, 1024, 16384, 1, 0, 0), (1024, 1024, 32768, 1, 0, 0),
    (512, 512, 512, 512, 1, 1), (512, 512, 512, 512, 0, 1), (1024, 1024, 768, 64, 1, 1), (4096, 4096, 4096, 8, 0, 0),
    (512, 512, 1024, 256, 0, 0), (512, 512, 1024, 256, 1, 1), (100, 128, 100000, 9, 0, 1),
]


# m, n, k, batch, op(A) / op(B) K-contiguous, both on the 16-byte grid, planes were the faster form
BF16X3 = [
    (64, 64, 4096, 1, 0, 0, 1, 1), (16, 16, 2048, 1, 0, 0, 1, 1), (2, 2000, 1024, 1, 0, 0, 1, 1), (2000, 2, 16384, 1, 0, 0, 1, 1),
    (512, 512, 16384, 1, 0, 0, 1, 1), (256, 256, 4096, 1, 0, 0, 1, 1), (128, 128, 1024, 1, 0, 0, 0, 1),
    (64, 512, 512, 1, 0, 0, 0, 1), (1024, 1024, 512, 1, 0, 0, 0, 1), (2048, 2048, 1024, 1, 0, 0, 0, 1),
    (1536, 1024, 4096, 1, 0, 0, 0, 1), (2048, 2048, 2048, 4, 0, 0, 0, 1), (2048, 2048, 2048, 4, 1, 1, 0, 1),
    (1000, 1000, 1000, 16, 1, 1, 0, 1), (300, 500, 2000, 64, 1, 1, 0, 1), (512, 512, 4096, 40, 1, 1, 0, 1),
    (64, 64, 512, 1, 0, 0, 1, 0), (512, 512, 1024, 1, 0, 0, 1, 0), (128, 4096, 4096, 1, 0, 0, 1, 0),
    (2048, 2048, 16384, 1, 0, 0, 1, 0), (1024, 1024, 2048, 1, 0, 0, 1, 0), (256, 256, 256, 256, 0, 0, 1, 0),
    (2048, 2048, 2048, 4, 1, 1, 1, 0), (512, 512, 4096, 40, 1, 1, 1, 0), (512, 512, 4096, 40, 0, 0, 0, 0),
    (300, 500, 2000, 64, 0, 0, 0, 0), (130, 130, 130, 1000, 0, 0, 0, 0), (128, 128, 1000, 300, 1, 1, 0, 0),
    (256, 256, 1000, 74, 1, 1, 0, 0), (512, 512, 512, 16, 0, 0, 0, 0),
    (992, 1072, 3136, 1, 1, 1, 1, 1), (592, 352, 2880, 2, 1, 0, 1, 1), (224, 80, 816, 4, 1, 0, 1, 1),
    (512, 112, 480, 2, 1, 1, 0, 1), (1664, 112, 7072, 3, 1, 1, 1, 0), (16, 1248, 448, 4, 0, 0, 1, 0), (1232, 2112, 1872, 6, 0, 1, 1, 0),
]
# parts, m, n, k, batch, form: 64 x 64, 128 x 64, 128 x 128, a pair
FORMS = [(3, 60, 50, 140, 3, 0), (3, 120, 150, 140, 2, 1), (3, 125, 127, 256, 140, 2), (3, 250, 255, 1000, 70, 3),
         (3, 1024, 1024, 1024, 16, 3), (3, 256, 256, 256, 256, 2), (3, 1024, 64, 512, 64, 1), (3, 1024, 1024, 1024, 1, 1),
         (2, 256, 256, 256, 256, 3), (2, 1024, 1024, 1024, 16, 3), (2, 64, 64, 10, 5, 0)]


def _check(tmp_path, call, rows):
    src = tmp_path / "t.cpp"
    src.write_text('#include "tile_rules.h"\n#include <cstdio>\nint main() {\n  const long r[][8] = {'
                   + ", ".join("{" + ", ".join(map(str, r)) + "}" for r in rows) + "};\n  int bad = 0;\n"
                   "  for (auto& x : r)\n    if (!(" + call + ")) std::printf(\"%ld %ld %ld %ld %ld\\n\", x[0], x[1], x[2], x[3],"
                   " x[4]), bad = 1;\n  if (!bad) std::puts(\"ok\");\n  return bad;\n}\n")
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(ROOT / "ssblasex_b200" / "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout)


def test_bf16x3_planes(tmp_path):
    _check(tmp_path, "ssb::bf16x3_planes(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[6], 148) == (x[7] != 0)", BF16X3)


def test_split_forms(tmp_path):
    _check(tmp_path, "ssb::split_form((int)x[0], x[1], x[2], x[3], x[4], 148).form == x[5]", FORMS)


def test_int8_tiles(tmp_path):
    rows = ", ".join("{%d, %d, %d, %d, %d, %d}" % r for r in I8)
    src = tmp_path / "t.cpp"
    src.write_text('#include "tile_rules.h"\n#include <cstdio>\nint main() {\n  const long r[][6] = {' + rows + '};\n'
                   '  for (auto& x : r)\n    if (ssb::i8_narrow_tiles(x[0], x[1], x[2], x[3], x[4] != 0, 148) != (x[5] != 0))'
                   ' return std::printf("%ld %ld %ld %ld\\n", x[0], x[1], x[2], x[3]), 1;\n  std::puts("ok");\n'
                   '  return 0;\n}\n')
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(ROOT / "ssblasex_b200" / "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout)
