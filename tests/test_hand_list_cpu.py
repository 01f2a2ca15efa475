"""The hand-over list's slots (csrc/pt_hand.h) when they run out: on the host, with
threads in the place of warps, and in the order of events in which giving a
range back loses records."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
ORDER = r'''
#include <cstdio>
#include "pt_hand.h"
/* 8 slots are left; 12, 4 and 4 are asked for.  (Given back, the first range lets
 * the third be written above the count that the second's return leaves.) */
int main()
{
    unsigned long long count = 32760;
    const unsigned asked[3] = { 12, 4, 4 };
    for (unsigned n : asked) {
        unsigned marks = 0;
        for (unsigned i = 0; i < n; ++i) marks += pt_hand_marks(count + i, 32768);
        std::printf("%d %u ", pt_hand_fits(count, n, 32768), marks);
        count += n;
    }
    std::printf("%llu %llu\n", pt_hand_written(count, 32768), pt_hand_written(32760, 32768));
}
'''


def _build(tmp_path, name, source):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = tmp_path / name
    subprocess.run([gxx, "-O2", "-std=c++17", "-pthread", "-I", str(ROOT / "particles_gb300" / "csrc"),
                    str(source), "-o", str(exe)], check=True)
    return exe


def test_every_written_slot_is_given_out_or_marked_once(tmp_path):
    exe = _build(tmp_path, "hand_check", ROOT / "tests" / "native" / "hand_check.cpp")
    r = subprocess.run([str(exe), "300", "8"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    given, marked, partial = (int(w) for w in r.stdout.split()[1::2])
    assert given + marked == 300 * 257 and given > 300 * 200 and 0 < partial <= 300


def test_a_warp_that_meets_the_end_marks_it(tmp_path):
    src = tmp_path / "order.cpp"
    src.write_text(ORDER)
    r = subprocess.run([str(_build(tmp_path, "order", src))], capture_output=True, text=True)
    assert [int(w) for w in r.stdout.split()] == [0, 8, 0, 0, 0, 0, 32768, 32760]
