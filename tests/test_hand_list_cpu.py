"""The hand-over list's slots (csrc/pt_hand.h) under concurrent reservations that
do not all fit: on the host, with threads in the place of warps, and step by
step through the order of events in which adding first and subtracting when
it did not fit loses records."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
ORDER = r'''
#include <cstdio>
#include "pt_hand.h"
/* A wants 12, B 4, C 4 of the 8 slots left; C and B act between A's first look
 * at the count and its answer. */
int main()
{
    unsigned long long count = 32760, c_at = 0, b_at = 0;
    auto cas = [&](unsigned long long e, unsigned long long w) {
        const unsigned long long was = count;
        if (was == e) count = w;
        return was;
    };
    auto slow = [&](unsigned long long e, unsigned long long w) {   /* the count moves on first */
        c_at = pt_hand_reserve(count, 4, 32768, cas);
        b_at = pt_hand_reserve(count, 4, 32768, cas);
        return cas(e, w);
    };
    const unsigned long long a_at = pt_hand_reserve(32760ull, 12, 32768, cas);
    const unsigned long long d_at = pt_hand_reserve(32760ull, 2, 32768, slow);
    std::printf("%llu %llu %llu %llu %llu\n", a_at, c_at, b_at, d_at, count);
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


def test_every_slot_below_the_count_is_given_out_once(tmp_path):
    exe = _build(tmp_path, "hand_check", ROOT / "tests" / "native" / "hand_check.cpp")
    r = subprocess.run([str(exe), "300", "8"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    given, refused = (int(w) for w in r.stdout.split()[1::2])
    assert given > 300 * 200 and refused >= 300 * 8


def test_a_reservation_that_does_not_fit_leaves_the_count_alone(tmp_path):
    src = tmp_path / "order.cpp"
    src.write_text(ORDER)
    r = subprocess.run([str(_build(tmp_path, "order", src))], capture_output=True, text=True)
    assert [int(w) for w in r.stdout.split()] == [32768, 32760, 32764, 32768, 32768]
