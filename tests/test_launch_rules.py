"""The launch rules of the cell chain (launch_rules.h, compiled for the host) against
measured times on a GB300 with 152 SMs, 48 hourly steps: the kernel of few cells or
the one of one thread a cell [horizons, cells, time of the first over time of the
second], and with outputs the latter's 4 or 3 blocks an SM [horizons, cells, time
with 4 over time with 3].  Where one is more than 3 % faster the rule takes it
(4 blocks: where they save a third of the waves); sizes on both sides of each line."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mhm_gb300" / "csrc"

LEAN, GENERAL, FLUX = "lean", "general", "flux"
MEASURED = {
    LEAN: [(1, 34040, .648), (1, 47524, .740), (1, 49506, 1.072), (1, 58322, 1.160), (1, 63001, 1.064), (1, 77562, 1.149),
           (2, 38025, .722), (2, 40804, .921), (2, 46656, .957), (2, 58322, 1.040), (2, 71824, 1.068), (2, 79524, 1.103),
           (3, 28561, .588), (3, 34969, .909), (3, 43681, .909), (3, 50850, .957), (3, 57600, 1.038), (3, 64009, 1.211),
           (4, 23716, .525), (4, 31506, .949), (4, 47961, .912), (4, 49729, 1.121), (5, 19044, .538), (5, 34040, .932),
           (5, 39800, 1.074), (6, 19044, .567), (6, 25281, .842), (6, 34040, .956), (6, 39800, 1.097), (7, 14280, .503),
           (7, 28730, .864), (7, 29756, 1.139), (8, 14280, .509), (8, 28730, .864), (8, 29756, 1.093)],
    GENERAL: [(1, 47524, .668), (1, 81796, .861), (1, 96100, .919), (1, 114921, 1.092), (2, 39601, .793), (2, 69960, .929),
              (2, 99856, .934), (2, 129960, 1.059), (3, 34969, .828), (3, 57600, .918), (3, 64009, 1.067),
              (3, 90000, 1.123), (4, 24806, .714), (4, 47961, .802), (5, 38416, .804), (5, 48620, .947), (6, 38416, .871),
              (6, 42642, .961), (7, 28730, .741), (7, 29756, .966), (7, 36480, 1.063), (8, 28730, .725), (8, 32041, .949)],
    # above 58,368 cells the other kernel's better number of blocks
    FLUX: [(1, 36864, .780), (1, 46656, 1.113), (1, 57840, 1.195), (1, 62500, 1.052), (1, 69960, 1.081), (1, 77006, 1.123),
           (1, 79806, .874), (1, 90000, .946), (1, 114921, 1.041), (1, 149769, 1.136), (2, 28561, .646), (2, 30625, 1.075),
           (2, 37830, 1.089), (2, 57840, 1.033), (2, 62500, 1.082), (2, 69960, 1.135), (2, 79806, .783), (2, 90000, .935),
           (2, 114921, 1.048), (2, 149769, 1.128), (3, 23716, .606), (3, 25440, .964), (3, 34040, 1.060), (3, 49729, 1.270),
           (3, 57840, 1.326), (3, 62500, 1.095), (3, 79806, .950), (3, 104976, 1.169), (4, 19740, .843), (4, 30976, .966),
           (4, 39800, 1.129), (4, 57840, 1.170), (4, 62500, 1.168), (4, 79806, .925), (4, 114921, 1.159), (5, 19740, .934),
           (5, 27225, 1.056), (5, 57840, 1.397), (5, 62500, 1.383), (5, 79806, 1.086), (6, 14280, .633), (6, 21756, .937),
           (6, 26896, 1.043), (6, 36480, 1.385), (6, 62500, 1.434), (7, 28730, .881), (7, 29756, 1.141), (7, 62500, 1.417),
           (7, 79806, 1.092), (8, 18906, .866), (8, 24180, .944)],
}
BLOCKS = [(1, 57840, 1.037), (3, 57840, 1.127), (5, 57840, 1.044), (8, 57840, 1.102), (1, 58564, .695), (5, 62500, .669),
          (6, 69960, .704), (8, 76729, .665), (2, 78400, 1.022), (3, 78400, 1.113), (5, 90000, 1.195), (8, 104976, 1.262),
          (1, 117992, .869), (5, 129960, .877), (8, 149769, .881), (4, 153664, .891), (3, 156816, 1.181),
          (8, 156816, 1.148), (1, 299756, .851), (5, 309692, .912), (8, 299756, .922)]
SRC = """#include "launch_rules.h"
extern "C" int small(int H, int lean, int flux, long long n, int sms) { return mhm::small_launch(H, lean, flux, n, sms); }
extern "C" int flux_blocks(long long n, int sms) { return mhm::flux_blocks_per_sm(n, sms); }
extern "C" int blocks(int H, int flux) { return mhm::small_blocks_per_sm(H, flux); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cc = shutil.which("g++") or shutil.which("c++")
    if not cc:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("rule")
    (d / "r.cpp").write_text(SRC)
    subprocess.run([cc, "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC), "-o", str(d / "r.so"), str(d / "r.cpp")], check=True)
    lib = C.CDLL(str(d / "r.so"))
    lib.small.argtypes = [C.c_int, C.c_int, C.c_int, C.c_longlong, C.c_int]
    lib.flux_blocks.argtypes = [C.c_longlong, C.c_int]
    return lib


def test_blocks_with_outputs(rule):
    assert not [p for p in BLOCKS if rule.flux_blocks(p[1], 152) != (4 if p[2] < 1 else 3)]
    for n in (1, 58368, 77825, 116736, 155649, 175104):
        assert rule.flux_blocks(n, 152) == 3
    for n in (58369, 77824, 116737, 155648, 291841):
        assert rule.flux_blocks(n, 152) == 4


@pytest.mark.parametrize("mode", [LEAN, GENERAL, FLUX])
def test_takes_the_faster_kernel(rule, mode):
    wrong = [p for p in MEASURED[mode]
             if abs(p[2] - 1) > 0.03 and bool(rule.small(p[0], mode == LEAN, mode == FLUX, p[1], 152)) != (p[2] < 1)]
    assert not wrong


def test_ends_and_other_gpus(rule):
    for H in range(1, 9):
        for lean, flux in ((1, 0), (0, 0), (0, 1), (1, 1)):
            assert rule.small(H, lean, flux, 1, 152)
            assert rule.small(H, lean, flux, 152 * rule.blocks(H, flux) * 32, 152)          # one full wave
            assert not rule.small(H, lean, flux, 10**7, 152) and not rule.small(H, lean, flux, 2**40, 152)
            # the lines follow the number of SMs
            for n in range(1000, 300000, 7777):
                assert rule.small(H, lean, flux, n * 152, 152) == rule.small(H, lean, flux, n * 76, 76)
    assert not rule.small(0, 1, 0, 1, 152) and not rule.small(9, 1, 0, 1, 152)
