"""The rule that gives small frames' marches four threads a pixel (csrc/gi_march_split.h)
against times measured on a GB300 (152 SMs): it chooses the faster form at sizes
where one is faster for the march and the two-bounce frame in every precision."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "gi_march_split.h"
#include <cstdio>
#include <cstdlib>
int main(int, char** v) {
  const int w = atoi(v[1]), h = atoi(v[2]), sub_w = (w + 3) / 4, sub_h = (h + 3) / 4;
  printf("%d", gi::split_pays(w, h, atoi(v[3]), (sub_w + 31) / 32 * ((sub_h + 3) / 4) * 16, 152));
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "split.cpp").write_text(PROGRAM)
    exe = d / "split"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'legitengine_gb300' / 'csrc'}", str(d / "split.cpp"), "-o",
                    str(exe)], check=True)
    return lambda *a: subprocess.run([str(exe)] + [str(v) for v in a], check=True, capture_output=True,
                                     text=True).stdout == "1"


@pytest.mark.parametrize("w,h,dirs", [(320, 240, 5), (400, 300, 4), (400, 300, 6), (400, 300, 7), (400, 300, 9),
                                      (400, 288, 6), (640, 480, 4), (640, 480, 6), (640, 480, 9), (960, 540, 8),
                                      (1280, 720, 12), (1920, 1080, 16)])
def test_one_thread_a_pixel_where_it_is_faster(split, w, h, dirs):
    assert not split(w, h, dirs)


@pytest.mark.parametrize("w,h,dirs", [(1, 1, 4), (256, 144, 4), (256, 144, 5), (256, 144, 32), (320, 180, 6),
                                      (320, 240, 8), (400, 288, 12), (512, 384, 8), (512, 384, 12), (640, 480, 16),
                                      (960, 540, 20)])
def test_four_threads_a_pixel_where_they_are_faster(split, w, h, dirs):
    assert split(w, h, dirs)
