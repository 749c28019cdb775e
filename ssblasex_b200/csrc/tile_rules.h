// Rules that choose a tile from the sizes of a call. Free of CUDA, so that they are tested on the CPU at the
// measured sides of each line.
#pragma once

namespace ssb {

// int8: whether a call takes 128 x 128 tiles (else 128 x 256). The wide tile reads a third less shared memory per
// product and is the faster one where the products bound the call (8 x 4096^3: 2570 TOPS against 1890); where
// bytes do, the narrow one is, whose shorter epilogues leave the memory idle for less. The line lies at 240
// operations per byte of operands and C, where neither leads by more than 10% (us, narrow and wide): beta = 1,
// 512 x 512^3 (102 per byte) 221, 257; 64 x (1024 x 1024 x 768) (162) 115, 129; 36 x (512 x 512 x 2048) (256)
// 35.5, 34.2; beta = 0, 512 x 512^3 (171) 136, 145; 192 x 640^3 (213) 90.9, 93.4; 256 x (512 x 512 x 768) (219)
// 85.7, 81.6; 128 x 768^3 (256) 91.4, 91.8; 256 x (512 x 512 x 1024) (256) 107, 96; 8 x 4096^3 (1365) 583, 429.
// Whatever the bytes, narrow tiles that fit one wave finish first, unless K is so long that the wide ones' K
// pieces fill more SMs than they do. Tiles of narrow / us narrow / us wide: k = 4096: 16 / 18.6 / 22.1,
// 96 / 15.2 / 23.0, 128 / 15.4 / 23.1, 192 / 25.5 / 16.7, 256 (2048^3: 15.9 / 12.4); k = 12288: 64 / 29.3 / 27.5,
// 96 / 35.3 / 34.8, 144 / 36.6 / 37.4; k = 16384: 32 / 24.5 / 28.4, 64 / 34.0 / 31.2, 128 / 45.9 / 41.8;
// k = 32768: 48 / 43.2 / 42.3, 64 / 54.6 / 43.6, 128 / 85.9 / 66.4.
inline bool i8_narrow_tiles(long m, long n, long k, long batch, bool read_c, long sms) {
  if (n <= 128) return true;
  const double ops = 2.0 * m * n * k, bytes = (double)m * k + (double)n * k + (read_c ? 8.0 : 4.0) * m * n;
  if (ops < 240.0 * bytes) return true;
  const double tiles = (double)((m + 127) / 128) * ((n + 127) / 128) * batch;
  return tiles <= sms && (k <= 12288 || 3 * tiles <= sms);
}

// The split kernel of the fp32 row (f32_split.cu): the tile whose waves end first, from the time of a chunk of
// 32 k and of a tile's end that each was measured to take (ns; fitted to 16 x 1024^3 and 4 x 2048^3, checked on 16
// other shapes). All give the same results bit for bit. Measured (us, 128 x 64 / 128 x 128 / a pair's 256 x 256):
// plain 16 x 1024^3 328 / 194 / 166, 256 x 256^3 98 / 62 / 74, 1 x 1024^3 32 / 34 / 47, 64 x (1024 x 64 x 512)
// 52 / 69 / 93; 3xBF16 16 x 1024^3 209 / 131 / 96, 256 x 256^3 65 / 44 / 39.
enum SplitForm { SPLIT_64, SPLIT_128_64, SPLIT_128_128, SPLIT_PAIR };
struct SplitChoice {
  SplitForm form;
  long waves;
  double ns;                 // its estimate
};
inline SplitChoice split_form(int parts, long m, long n, long k, long batch, long sms) {
  struct Cost {
    long tm, tn, ctas, chunk, tile;
  };
  const Cost plain[4] = {{64, 64, 1, 750, 300}, {128, 64, 1, 750, 300}, {128, 128, 1, 780, 2600}, {256, 256, 2, 1030, 8500}};
  const Cost bf16x3[4] = {{64, 64, 1, 445, 1500}, {128, 64, 1, 430, 1100}, {128, 128, 1, 520, 2100}, {256, 256, 2, 610, 4400}};
  const long nkc = (k + 31) / 32;
  SplitChoice best{SPLIT_64, 0, 0.0};
  const bool small = m <= 64 && n <= 64;
  for (int i = small ? 0 : 1; i < (small ? 1 : 4); ++i) {
    const Cost& c = (parts == 3 ? plain : bf16x3)[i];
    const long tiles = (m + c.tm - 1) / c.tm * ((n + c.tn - 1) / c.tn) * batch, workers = sms / c.ctas;
    const long waves = (tiles + workers - 1) / workers;
    const double t = (double)waves * (double)(nkc * c.chunk + c.tile);
    if (best.waves == 0 || t < best.ns) best = {(SplitForm)i, waves, t};
  }
  return best;
}

// 3xBF16: whether a call takes the split pass and the tiled GEMM over its planes, else the split kernel, whose results
// are the same bits. The split kernel saves the planes' 8 bytes per element, but a chunk of 32 k takes it longer than the
// tiled GEMM: where the tiles are few that is most of the call, and more so where the operands are off the
// 16-byte grid (its converters then copy 4 bytes at a time) or tiles are part-filled. Estimates in ns, from
// launches, chunks and the planes at the rate that the pass reaches by layout. Measured (us, split kernel / planes),
// aligned: 64 x 64 x 4096 62 / 47, 512 x 512 x 16384 245 / 201, 2 x 2000 x 4096 108 / 69, 992 x 1072 x 3136 78 / 52,
// 1024 x 1024 x 16384 246 / 245, 2048 x 2048 x 4096 86 / 134, 40 x (512 x 512 x 4096) 255 / 657; off the grid: 128 x 128
// x 1024 37 / 20, 1536 x 1024 x 4096 172 / 78, 4 x 2048^3 NT 346 / 244, TN 384 / 223, 16 x 1000^3 NT 181 / 195,
// 300 x (128 x 128 x 1000) 134 / 272; short K: 512 x 112 x 480 23 / 18, 1536 x 1024 x 256 off the grid 17 / 16,
// 1000 x 130^3 113 / 233.
inline bool bf16x3_planes(long m, long n, long k, long batch, bool a_kcontig, bool b_kcontig, bool a_on_grid,
                          bool b_on_grid, long sms) {
  if (k < 384) return false;
  const SplitChoice c = split_form(2, m, n, k, batch, sms);
  const long rows = c.form == SPLIT_64 ? 64 : c.form == SPLIT_PAIR ? 256 : 128;
  const long cols = c.form == SPLIT_PAIR ? 256 : c.form == SPLIT_128_128 ? 128 : 64;
  // how much longer a chunk takes: half and thin tiles, ragged edges (of a single wave, the longest tile counts),
  // operands off the grid
  double slower = 1.06;
  if (m <= rows / 2 || n <= cols / 2) slower = c.form != SPLIT_64 && (m <= rows / 8 || n <= cols / 8) ? 1.75 : 1.45;
  else if (m % rows || n % cols) slower = c.waves > 1 ? 1.25 : m % rows ? 1.7 : 1.3;
  const double off = c.form == SPLIT_64 ? 0.25 : 0.5;
  const double grid = 1.06 + (a_on_grid ? 0.0 : off + (a_kcontig ? 0.15 : 0.0)) + (b_on_grid ? 0.0 : off + (b_kcontig ? 0.25 : 0.0));
  if (grid > slower) slower = grid;
  const double split = 4000.0 + c.ns * slower;
  const long bn = n <= 64 ? 64 : 128, tiles = (m + 127) / 128 * ((n + bn - 1) / bn) * batch;
  const double pass = 8.0 * (double)k * (double)batch * ((double)m / (a_kcontig ? 4200.0 : 3100.0) +
                                                        (double)n / (b_kcontig ? 4200.0 : 3100.0));
  const double planes = 9000.0 + pass + (double)((tiles + sms - 1) / sms) *
                                            ((double)((k + 31) / 32) * (bn == 64 ? 290.0 : 330.0) + 2500.0);
  return planes < split;
}

}  // namespace ssb
