// gi_march_split.h -- when a whole frame's march takes the direction split (four threads a
// pixel, gi_march.cu): plain C++.
#pragma once

namespace gi {

constexpr int kSplit = 4;  // threads of a pixel, each with every fourth of its directions

// Whether an untuned frame of the standard form takes the direction split: four times the
// threads, each with the pixel's set-up and up to n = ceil(R / 4) of its directions.  It
// pays while the one-thread form is too few waves of CTAs (8 an SM) to fill the GPU and
// hide its latency, and up to more waves the more directions share the set-up and the
// more evenly they divide.
//
// The line, (1.5 n - 1) waves times the share of the last round of directions that is
// used, follows sweeps of 256 x 144 to 1600 x 900 with 4 to 32 directions.  One-thread
// form / split in us, march and two-bounce frame, steps capped at 64:
//   exact    R =  8   256 x 144 (0.24 waves)   108 / 55      190 / 120
//                     512 x 384 (1.3)          240 / 208     368 / 338
//                     640 x 480 (2.0)          324 / 311     483 / 485
//                     700 x 500 (2.2)          387 / 383     568 / 580
//                     1600 x 900 (9.3)        1289 / 1402   1785 / 2019
//            R = 16   960 x 540 (3.3)         1562 / 1491   2089 / 2025
//                     1280 x 720 (5.9)        2538 / 2507   3314 / 3382
//            R =  4   320 x 240 (0.49)          54 / 49      118 / 113
//                     400 x 300 (0.77)          61 / 71      131 / 148
//   texture  R =  5   256 x 144                 32 / 26       99 / 83
//            R =  8   640 x 480                137 / 137     295 / 303
// One line serves the three precisions: over 27 sizes with up to 16 direction counts each,
// what it splits is at most 6 % slower for it (8 % at 400 x 300).
// Five directions, whose second round leaves three of a pixel's threads idle, stop
// earlier: at 320 x 240 (0.49 waves) exact 72 / 72 and 142 / 144, fast 48 / 52 and 121 /
// 126, texture 40 / 42 and 109 / 112.
// CTAs that just fill the GPU once run best in the one-thread form: at 400 x 300 (one full
// wave, its ragged tiles included) and R = 6, 7 and 9 exact 106 / 124, 132 / 142 and 188 /
// 212, texture 52 / 63, 59 / 68 and 77 / 91, frames 134 / 151, 150 / 162 and 193 / 205; there the
// split needs 8 directions in even rounds (exact 160 / 162, frame 270 / 265) or 13.
//
// tiles: CTAs of the one-thread form in 4 rows (32 x 4 pixels of a pattern each).
inline bool split_pays(int width, int height, int dirs, int tiles, int sms) {
  const int n = (dirs + kSplit - 1) / kSplit, full = 8 * sms;
  const float waves = (float)width * (float)height / (128.0f * (float)full);
  const float line = dirs == 5 ? 0.45f : (1.5f * (float)n - 1.0f) * (float)(dirs - kSplit * (n - 1)) / (float)kSplit;
  const bool one_full_wave = tiles <= full && 10ll * tiles > 9ll * full;
  if (one_full_wave && line < 2.0f && n < 4) return false;
  return waves < line;
}

}  // namespace gi
