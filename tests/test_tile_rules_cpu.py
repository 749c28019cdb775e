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
