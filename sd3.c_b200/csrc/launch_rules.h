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

}  // namespace sd3
