"""log / exp / pow at the seams of their main paths: arguments next to the
multiples of ln2/128 and to the table's interval ends, where a reduction can
come out on either side, and next to the ends of the ranges the main paths
take -- within 1 ulp of the C library, on the host and on the device."""
import ctypes as C

import numpy as np
import pytest

_dp = C.POINTER(C.c_double)
LN2_128 = np.log(2.0) / 128


def _around(x, rng, bits=52):
    """x and neighbours of x at every relative distance down to the last bit."""
    d = np.exp2(-rng.uniform(8, bits + 1, x.size)) * rng.choice([-1.0, 1.0], x.size)
    return np.concatenate([x, x * (1 + d), np.nextafter(x, np.inf), np.nextafter(x, -np.inf)])


def _cases(rng):
    k = rng.integers(1, 130_000, 60_000)
    ex = _around(k * LN2_128, rng)
    ends = np.array([2.0**-8, 708.0, 707.999])
    exp = np.concatenate([ex[ex < 709], -ex[ex < 745], _around(ends, rng), -_around(ends, rng)])
    with np.errstate(over="ignore"):
        z = (1 + np.arange(257) / 256.0)[:, None] * np.exp2(np.array([-1022.0, -300, -30, -2, -1, 0, 1, 40, 1023]))
    x = _around(z[np.isfinite(z)].reshape(-1).repeat(20), rng)
    log = np.concatenate([x[(x > 0) & np.isfinite(x)], _around(np.array([1 - 2.0**-7, 1 + 2.0**-7, 1.0]), rng)])
    y = rng.uniform(2.0**-10, 2.0, 60_000)
    y[:6] = [2.0**-10, np.nextafter(2.0, 0), 2.0, 1.0, 2 / 3, 0.5]
    with np.errstate(over="ignore"):
        px = _around(np.exp2(rng.integers(-10_000, 10_000, y.size) / 128.0 / y), rng)
    py = np.tile(y, 4)
    ok = (px > 0) & np.isfinite(px)
    return log, exp, px[ok], py[ok]


@pytest.mark.parametrize("where", [0, pytest.param(1, marks=pytest.mark.gpu)])
def test_seams(lib, where):
    log, exp, px, py = _cases(np.random.default_rng(4))
    with np.errstate(over="ignore", under="ignore"):
        for op, x, y, ref in ((0, log, None, np.log(log)), (1, exp, None, np.exp(exp)), (2, px, py, np.power(px, py))):
            x = np.ascontiguousarray(x)
            out = np.empty_like(x)
            rc = lib.mhm_hmath_eval(op, where, x.size, x.ctypes.data_as(_dp),
                                    None if y is None else np.ascontiguousarray(y).ctypes.data_as(_dp),
                                    out.ctypes.data_as(_dp))
            assert rc == 0
            d = np.abs(out.view(np.int64) - ref.view(np.int64))
            assert d.max() <= 1, (op, x[d.argmax()], out[d.argmax()], ref[d.argmax()])
