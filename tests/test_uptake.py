"""hm_uptake (fp64i.h), a horizon's uptake on the integer pipe, against the five
FP64 operations it stands for (src/mHM/mo_soil_moisture.f90:254-286 with the
Feddes stress of :358), compiled for the host: where it takes the operands, the
evapotranspiration and the storage left are theirs bit for bit; what it cannot
do it refuses."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "mhm_gb300" / "csrc"

SRC = r"""
#include "hmath.h"
#include "fp64i.h"
/* taken[i] (with r, left), and the FP64 operations' r0, left0 */
void uptake(long n, const double *S, const double *pw, const double *fc, const double *f, const double *a,
            int *taken, double *r, double *left, double *r0, double *left0)
{
    for (long i = 0; i < n; ++i) {
        const double den = fc[i] - pw[i];
        const int wet = S[i] >= fc[i];
        volatile double t = f[i];
        if (!wet) {
            volatile double d = S[i] - pw[i];
            t = f[i] * d;
            t = t / den;
        }
        volatile double x = a[i] * t, y = S[i] - x;
        r0[i] = x;
        left0[i] = y;
        r[i] = left[i] = -1.0;
        taken[i] = hm_uptake(S[i], pw[i], f[i], a[i], wet, hm_recip_of(den), (int)(hm_hi(hm_d2b(den)) >> 20),
                             &r[i], &left[i]);
    }
}
int in_range(double x) { return hm_uptake_var(x); }
"""


@pytest.fixture(scope="module")
def uptake(tmp_path_factory):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("uptake")
    (d / "u.c").write_text(SRC)
    subprocess.run([cc, "-O2", "-std=c99", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(CSRC), "-o", str(d / "u.so"),
                    str(d / "u.c"), "-lm"], check=True)
    lib = C.CDLL(str(d / "u.so"))
    lib.in_range.argtypes = [C.c_double]

    def run(S, pw, fc, f, a):
        n = S.size
        ins = [np.ascontiguousarray(x, np.float64) for x in (S, pw, fc, f, a)]
        taken = np.zeros(n, np.int32)
        outs = [np.zeros(n) for _ in range(4)]
        p = lambda x: x.ctypes.data_as(C.c_void_p)   # noqa: E731
        lib.uptake(C.c_long(n), *map(p, ins), p(taken), *map(p, outs))
        return taken != 0, *outs
    run.in_range = lib.in_range
    return run


def _soil(rng, n):
    """Wilting point, field capacity (2^-4 <= FC - PW < 2^11, as the kernel asks
    before it comes here), root fraction and demand of a horizon."""
    pw = 10.0 ** rng.uniform(-3, 3, n)
    fc = pw + np.exp2(rng.uniform(-3.9, 10.9, n))
    return pw, fc, rng.uniform(0.001, 1.0, n), 10.0 ** rng.uniform(-9, 1, n)


def _check(uptake, S, pw, fc, f, a):
    """the kernel's conditions; returns what was taken and the true uptake"""
    ok = (S > pw) & (S >= 2.0**-50) & (fc - pw >= 2.0**-4) & (fc - pw < 2.0**11)
    S, pw, fc, f, a = (x[ok] for x in (S, pw, fc, f, a))
    taken, r, left, r0, left0 = uptake(S, pw, fc, f, a)
    same = (r.view(np.uint64) == r0.view(np.uint64)) & (left.view(np.uint64) == left0.view(np.uint64))
    bad = np.flatnonzero(taken & ~same)
    assert bad.size == 0, [x[bad[0]].hex() for x in (S, pw, fc, f, a, r, r0, left, left0)]
    assert not (taken & (r0 >= 0.5 * S)).any()          # more than half of the store: refused
    assert not (taken & (S < fc) & (S >= 4096.0 * pw)).any()   # dry, more than 2^11 apart: refused
    untouched = ~taken
    assert (r[untouched] == -1.0).all() and (left[untouched] == -1.0).all()
    return taken, S, fc, r0


@pytest.mark.parametrize("seed", range(3))
def test_ordinary_soils(uptake, seed):
    rng = np.random.default_rng(seed)
    pw, fc, f, a = _soil(rng, 400_000)
    S = pw + (fc - pw) * rng.uniform(0.0, 1.6, pw.size)     # dry and wet
    taken, S, fc, r0 = _check(uptake, S, pw, fc, f, a)
    small = (r0 < 0.25 * S) & (r0 > S * 2.0**-58)
    assert (S >= fc).any() and (S < fc).any()
    # refused of these only dry soils 2^11 apart and the roundings left open (one in 512)
    assert taken[small & (S >= fc)].all()
    assert taken.mean() > 0.7


def test_next_to_the_wilting_point_and_the_field_capacity(uptake):
    rng = np.random.default_rng(5)
    pw, fc, f, a = _soil(rng, 200_000)
    eps = np.exp2(-rng.uniform(1, 53, pw.size))
    for S in (pw * (1 + eps), np.nextafter(pw, np.inf), fc * (1 - eps / 4), np.nextafter(fc, 0), fc, np.nextafter(fc, np.inf)):
        taken = _check(uptake, S, pw, fc, f, a * np.exp2(rng.uniform(-20, 0, pw.size)))[0]
        assert taken.any()


def test_ties(uptake):
    """Short mantissas: products, differences and quotients that are exact, or
    lie halfway between two doubles."""
    rng = np.random.default_rng(6)
    n = 400_000

    def short(bits, lo, hi):
        return rng.integers(1 << (bits - 1), 1 << bits, n) * np.exp2(rng.integers(lo, hi, n) - bits)
    pw = short(8, 0, 8)
    fc = pw + short(6, -2, 10)
    f = short(27, -4, 1)
    a = short(27, -12, 4)
    for S in (pw + short(12, -6, 10), fc + short(20, -3, 6), short(53, 2, 11)):
        taken = _check(uptake, S, pw, fc, np.minimum(f, 1.0), a)[0]
        assert taken.any()


def test_edges_of_the_ranges(uptake):
    for x, want in ((2.0**-200, 1), (np.nextafter(2.0**-200, 0), 0), (np.nextafter(2.0**200, 0), 1), (2.0**200, 0), (0.0, 0),
                    (-1.0, 0), (np.inf, 0), (-np.inf, 0), (np.nan, 0), (5e-324, 0)):
        assert bool(uptake.in_range(x)) == bool(want), x
    # demands and root fractions down to 2^-200: the uptake is too small for 64 bits, or exact
    rng = np.random.default_rng(7)
    pw, fc, f, a = _soil(rng, 100_000)
    S = pw + (fc - pw) * rng.uniform(0.0, 1.6, pw.size)
    _check(uptake, S, pw, fc, f * np.exp2(-rng.uniform(0, 190, pw.size)), a)
    _check(uptake, S, pw, fc, f, np.exp2(rng.uniform(-200, 199, pw.size)))
    _check(uptake, S * np.exp2(rng.uniform(0, 180, pw.size)), pw, fc, f, a * np.exp2(rng.uniform(0, 180, pw.size)))
