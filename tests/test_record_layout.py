"""The march record's offsets (csrc/gi_record.h) at the sizes a record can have, on the
CPU: rows and blocks lie one after the other, and the last one ends at the record's
length.  Products of 2^32 and more are in reach (9216 x 8192 with 59 steps, 12288 x 9216
with 41), where 32-bit offsets would lay one pixel's values over another's."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "gi_record.h"
#include <cstdio>
#include <cstdlib>
int main(int, char** v) {
  const int w = atoi(v[1]), h = atoi(v[2]), p = atoi(v[3]), dirs = atoi(v[4]), steps = atoi(v[5]);
  const size_t npix = gi::record_pixels(w, h, p);
  printf("%zu\n", npix);
  for (int d = 0; d < dirs; d++)
    for (int s = 0; s < steps; s++)
      printf("%zu\n", gi::record_block(d, steps, (unsigned)npix) + gi::record_row(s, (unsigned)npix));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("record")
    (d / "record.cpp").write_text(PROGRAM)
    exe = d / "record"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'legitengine_gb300' / 'csrc'}", str(d / "record.cpp"), "-o",
                    str(exe)], check=True)
    return exe


@pytest.mark.parametrize("w,h,pattern,dirs,steps", [
    (1, 1, 1, 1, 1), (33, 17, 4, 3, 24), (1920, 1080, 4, 16, 64), (9216, 8192, 4, 1, 59), (12288, 9216, 4, 1, 41),
    (12288, 9216, 4, 3, 59), (46340, 46340, 1, 4, 64)])
def test_rows_follow_each_other(program, w, h, pattern, dirs, steps):
    out = subprocess.run([str(program)] + [str(v) for v in (w, h, pattern, dirs, steps)], check=True,
                         capture_output=True, text=True).stdout.split()
    npix, rows = int(out[0]), [int(v) for v in out[1:]]
    up = lambda n: -(-n // pattern)
    assert npix == pattern * pattern * up(w) * up(h) and npix < 2 ** 31
    assert rows == [npix * k for k in range(dirs * steps)]
