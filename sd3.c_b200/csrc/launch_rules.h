// Which of several kernels that give the same bits a size runs on, by what was measured on both sides of each line.
// Plain C++, so that the lines can be checked on the host.
#pragma once

namespace sd3 {

// LayerNorm + modulate, by row width E, rows of the launch (both problems) and whether a problem has two modulations.
//   LN_WARP_PER_ROW   a warp per row, 2, 6 or 12 quads a lane by the width, modulation vectors staged in shared memory
//   LN_CTA_PER_ROW    four warps per row, which always go through 12 quads a lane: rows of up to 1536
//   LN_ROWS_PER_CTA   the same with several consecutive rows, whose modulation vectors stay in registers
enum LnKernel { LN_WARP_PER_ROW, LN_CTA_PER_ROW, LN_ROWS_PER_CTA };
constexpr int LN_ROW_QUADS = 12;
// us, a warp per row / the kernel that the rule takes (in brackets: the one that it does not take):
//   one modulation                                     two modulations
//   E  256    450 rows  2.10 /  1.96                    450 rows   2.18 / (2.51)
//             888 rows  2.12 / (2.80)                  4429 rows   3.21 / (6.76)
//           35432 rows 11.1  / (35.8)                 35432 rows  14.6  / (42.7)
//   E  768    450 rows  2.83 /  2.10                    450 rows   3.54 /  2.72
//             888 rows  2.87 / (3.11)                   888 rows   3.56 / (3.66)
//           35432 rows 29.0  / (42.6)                 35432 rows  40.2  / (54.4)
//   E 1024   1357 rows  4.46 /  3.65                   4429 rows  10.2  /  7.94
//            8858 rows 11.2  / (14.0)                 35432 rows  73.5  / 60.5
//           17000 rows 23.7  / (24.3)
//   E 1280   8858 rows 12.8  / (14.8)                  4429 rows  11.6  /  8.34
//            9500 rows 21.5  /  15.2                  35432 rows  85.8  / 69.8
//   E 1536   1357 rows  5.31 /  3.96                    589 rows   6.70 /  3.06
//            4429 rows  8.34 / (8.95)                  1357 rows   8.26 /  4.08
//            8200 rows 14.6  /  12.3 (x in L2), 18.8 / 14.1 (x in HBM); 8858 rows 14.9 / 15.6, 19.5 / 18.8
//           13287 rows 29.0  /  23.5                  13287 rows  47.5  / 30.1
//           35432 rows 60.6  /  55.2                  35432 rows  97.4  / 76.0
inline LnKernel ln_kernel(int E, long rows, bool dual, int sms) {
  if (E > 4 * 32 * LN_ROW_QUADS) return LN_WARP_PER_ROW;
  if (rows <= 4L * sms) return !dual ? LN_CTA_PER_ROW : E > 256 ? LN_ROWS_PER_CTA : LN_WARP_PER_ROW;
  if (E <= 768) return LN_WARP_PER_ROW;
  if (dual) return LN_ROWS_PER_CTA;
  if (rows <= 3700) return LN_CTA_PER_ROW;
  // up to 64 rows an SM the warps take two rows each in one wave
  return (E > 1280 ? rows > 8000 : E > 1024 && rows > 64L * sms) ? LN_ROWS_PER_CTA : LN_WARP_PER_ROW;
}

// Width of a CTA-pair GEMM's tiles (256 rows each): the one with the least time by waves of `pairs` CTA pairs.  A wave of
// 128-wide tiles takes 0.64 of a wave of 256-wide ones (half the MMA time, but 96 bytes of operands per clock and SM where
// TMA brings at most 82 to 92), and the last wave's epilogue, which nothing overlaps, is half as long, worth about ten
// K blocks of a wide tile, less where K (in elements) is so short that the epilogues set the pace: 0.4 blocks per
// 64 of K.  A K block is 64 of K in bf16, 128 in e4m3.  Measured, us, wide / narrow (waves of each):
//   K 1536, QKV    589 rows 15.0 / 12.9 (1, 2)   1357: 21.7 / 18.5 (2, 3)   2714: 30.3 / 33.3 (3, 6)   4429: 49.1 / 52.2 (5, 9)
//   K 1536, GELU   333 rows 15.8 / 13.3 (1, 2)   1024: 21.0 / 19.1 (2, 3)   1357: 23.7 / 24.7 (2, 4)   4429: 61.9 / 71.7 (6, 12)
//   K 1536, gate  2714 rows 14.5 / 14.6 (1, 2)   4429: 23.5 / 21.2 (2, 3)   5428: 26.7 / 28.8 (2, 4)
//   K 4096, fp32 output (the captions)  333 rows 24.8 / 14.9 (1, 1)   1332: 25.2 / 16.0 (1, 1)
//   K 6144, gate  2714 rows 38.6 / 43.6 (1, 2)   4429: 68.8 / 67.4 (2, 3)   5428: 75.4 / 86.9 (2, 4)
//   K 1024, N 1024, gate 8192 rows 17.6 / 19.3 (2, 4)   16384: 34.1 / 37.3 (4, 7)   GELU 16.1 / 18.1, 27.4 / 31.7
//   K 512, N 512, gate 16384 rows 13.1 / 14.1 (2, 4)   N 1536, bias 8192 rows 13.2 / 14.8 (3, 6)
// (an FP8 dual block of width 1536, 576 + 333 tokens, whose QKV and MLP1 launches are both (2, 4): 105 us with ten blocks, 109
// with 4.8)
// after256: those of the 256-wide tiles that run after another one on the same pair (pair_tiles.h), a wave of their own.
// gate: the gate + residual GEMMs, the ones with few tiles, have 64-wide ones too, for problems that fit one wave of
// those.  us, 128 / 64 wide: K 6144, 256 rows 19.7 / 17.9, 333 rows 19.8 / 18.5, 700 rows 19.9 / 19.5; K 1536, 256 rows
// 7.7 / 7.0, 589 rows 8.2 / 8.2 (slots of four stages: 20.1 at 256 rows).
inline int pair_tile_width(long tiles256, long after256, int K, bool fp8, bool gate, int pairs) {
  if (pairs <= 0) return 256;
  const long first256 = tiles256 - after256;
  if (gate && 4 * first256 <= pairs) return 64;
  const long wide = (first256 + pairs - 1) / pairs + (after256 + pairs - 1) / pairs;
  const long narrow = (2 * first256 + pairs - 1) / pairs + (2 * after256 + pairs - 1) / pairs;
  const long k64 = (K + 63) / 64, k_blocks = fp8 ? (k64 + 1) / 2 : k64;
  const long epilogue = 40 * k64 < 1000 ? 40 * k64 : 1000;  // in hundredths of a wide tile's K block
  return 64 * narrow * k_blocks < 100 * wide * k_blocks + epilogue ? 128 : 256;
}

}  // namespace sd3
