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

}  // namespace ssb
