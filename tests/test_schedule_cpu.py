"""The host arithmetic that shapes the launches (csrc/schedule.h), compiled as it is and compared with plain searches."""
import ctypes
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "flash-triangle-attention_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("schedule")
    src = d / "schedule.cpp"
    src.write_text('#include "schedule.h"\n'
                   'extern "C" int fwd_grid_rows(int n, long long per, int sms) { return fta::fwd_grid_rows(n, per, sms); }\n')
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(d / "s.so")], check=True)
    s = ctypes.CDLL(str(d / "s.so"))
    s.fwd_grid_rows.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int]
    return s


def _search(ngroups, per, sms):
    """Every grid.y up to 96, or up to what one wave holds."""
    most = min(ngroups, max(96, sms // per))
    eff = [per * ngroups / (-(-per * gy // sms) * sms * (-(-ngroups // gy) + 0.35)) for gy in range(1, most + 1)]
    return 1 + next(i for i, e in enumerate(eff) if e >= 0.97 * max(eff))


def test_forward_grid_is_that_of_a_plain_search(lib):
    # one (query block, head) pair: a wave has room for 148 CTAs of it
    assert lib.fwd_grid_rows(512, 1, 148) == 128  # 1024 rows in groups of two: four groups each, not six
    assert lib.fwd_grid_rows(256, 1, 148) == 128  # in groups of four
    assert lib.fwd_grid_rows(148, 1, 148) == 148
    assert lib.fwd_grid_rows(148, 3, 148) == 37   # one wave, not three of the shortest CTAs
    assert lib.fwd_grid_rows(192, 24, 148) == 6   # B1 H4 L768 D32
    rng = random.Random(5)
    shapes = [(n, per) for n in range(1, 40) for per in (1, 2, 3, 7, 24, 147, 148, 149)]
    shapes += [(rng.randint(1, 1100), rng.choice([1, 2, 3, 4, 8, 12, 16, 24, 48, 64, 128, 256, 1000])) for _ in range(400)]
    for n, per in shapes:
        assert lib.fwd_grid_rows(n, per, 148) == _search(n, per, 148), (n, per)
