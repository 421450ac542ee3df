"""A node above the tiles counts as written when both of its corners say so: never for cleared padding, whatever the
other corner holds, in any build; and what it carries comes back."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "climb_message.h"
using namespace bvhgb;
int main() {
  for (uint64_t e = 64; e < (1ull << 32); e += 64) {  // every epoch
    const uint32_t epoch = (uint32_t)e, mark = climb_mark(epoch);
    if (mark == 0 || mark > 0xffffu) return 1;
    const uint32_t w = climb_hi_word(mark, (uint32_t)(e >> 6) & 255u, (uint32_t)(e >> 14) & 255u);
    if (!climb_whole(epoch, w, epoch, mark)) return 2;
    if (climb_whole(epoch, 0, epoch, mark)) return 3;  // the lower corner is there, the upper is not
    if (climb_whole(0, w, epoch, mark)) return 4;      // the upper corner is there, the lower is not
    if (climb_delta(w) != ((e >> 6) & 255u) || climb_height(w) != ((e >> 14) & 255u)) return 5;
    // a corner of the build before, of this build's neighbours in the 16-bit count, of any other epoch
    const uint32_t other = epoch - 64, far = epoch ^ 65536u * 64u;
    if (climb_whole(other, w, epoch, mark) || climb_whole(far, w, epoch, mark)) return 6;
    if (climb_whole(epoch, climb_hi_word(climb_mark(other), 0, 0), epoch, mark)) return 7;
  }
  for (uint32_t h = 255; h < 600; ++h)
    if (climb_height(climb_hi_word(1, 0, h)) != 255u) return 8;
  puts("ok");
}
"""


def test_messages(tmp_path):
    src = tmp_path / "m.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "m"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", os.path.join(ROOT, "bvh_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "ok\n")
