"""The ends of the exponent range in the FP64 form's fixed-point transforms (fft_fx.cuh), restated on the CPU
in exact integers: rows of every finite scale, denormal ones among them, enter on one exponent
and leave as doubles of the result's own exponent.

The stages are test_fx_algorithm's; here are the scale of a row, its elements' way in and the results' way
out as the kernel has them.  Bound: 2^-53 of the result's 2-norm for the integers (as there), half a unit of
the last place for each result's rounding, and below the normal range two half units of the smallest
denormal (the rounding to 53 bits comes first)."""
import math

import numpy as np
import pytest

from test_fx_algorithm import dft_ld, l1, stages

EMIN, EB_MIN, EB_MAX, BITS = 96, 64, 2045, 59


def bits(d):
    return int(np.float64(d).view(np.uint64))


def field(d):
    return (bits(d) >> 52) & 0x7ff


def from_double(d, em):
    """fx_from: the leading bit is taken for set, and the shift is an unsigned difference."""
    b = bits(d)
    s = min((em - field(d)) % 2**32, 63)
    m = (b & (2**52 - 1)) | 2**52
    v = (((m << (BITS - 52)) >> s) + 1) >> 1
    return -v if b >> 63 else v


def enter(row):
    """fx_scale and fx_enter of the components: (integers, exponent field of the scale)."""
    em = min(max(max(field(d) for d in row), 1), 2046)
    if em >= EMIN:
        return [from_double(d, em) for d in row], em
    return [from_double(d * 2.0**128, em + 128) if d != 0.0 else 0 for d in row], em


def leave(q, e):
    """fx_leave: fx_to with the exponent in its range, then a power of two."""
    b = e + 63 + 1022
    eb = min(max(b, EB_MIN), EB_MAX)
    out = []
    for v in q:
        m = abs(v)
        if m == 0:
            out.append(0.0)
            continue
        lz = 64 - m.bit_length()
        n = (m << lz) % 2**64
        w = (n >> 11) + ((n >> 10) & 1) + ((eb - lz) << 52)
        assert 2**52 <= w < 2047 * 2**52, "outside the normal range"
        d = float(np.uint64(w).view(np.float64))
        with np.errstate(over="ignore", under="ignore"):
            out.append(math.copysign(float(np.float64(d) * np.float64(2.0)**(b - eb)), v))
    return np.array(out)


SCALES = [2.0**-1074, 3e-320, 2.0**-1030, 1e-308, 1e-305, 1e-300, 1e-290, 1e-280, 2.0**-930, 2.0**-928, 2.0**-927, 2.0**-926,
          1.0, 2.0**1005, 2.0**1006, 2.0**1007, 2.0**1013]


@pytest.mark.parametrize("scale", SCALES)
def test_rows_of_every_scale(scale):
    n = 64
    rng = np.random.default_rng(5)
    rows = {"noise": rng.standard_normal(n) + 1j * rng.standard_normal(n),
            "wide": (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 10.0 ** rng.uniform(-18, 0, n),
            "spike": np.where(np.arange(n) == 21, 1.0 + 0.5j, 0.0)}
    for name, z in rows.items():
        z = z / max(np.abs(z.real).max(), np.abs(z.imag).max()) * scale  # rounded to what the type holds
        c = np.concatenate([z.real, z.imag])
        q, em = enter(c)
        assert max(abs(v) for v in q) <= 2**BITS
        v, d = stages(list(zip(q[:n], q[n:])), False, BITS, True, sum(l1(a) for a in q))
        e = em - 1022 - BITS + d
        got = leave([a for a, _ in v], e), leave([b for _, b in v], e)
        ref = dft_ld(z.astype(np.clongdouble), -1)
        nrm = np.sqrt(ref[0]**2 + ref[1]**2)
        err = np.sqrt((got[0] - ref[0])**2 + (got[1] - ref[1])**2)
        norm = np.sqrt((nrm**2).sum()) if scale > 1e-300 else nrm.max() * np.sqrt(np.longdouble(n))
        tiny = np.longdouble(2.0)**-1074
        assert np.isfinite(got).all(), name
        assert (err <= 2 * np.longdouble(2.0)**-53 * norm + 2 * tiny).all(), (name, float((err / (norm + tiny)).max()))


def test_results_beyond_the_largest_double_are_infinite():
    n = 16
    z = np.full(n, 2.0**1023)
    q, em = enter(np.concatenate([z, np.zeros(n)]))
    v, d = stages(list(zip(q[:n], q[n:])), False, BITS, True, sum(l1(a) for a in q))
    got = leave([a for a, _ in v], em - 1022 - BITS + d)
    assert got[0] == np.inf and not got[1:].any()


def test_zero_rows_stay_zero():
    q, em = enter(np.array([0.0, -0.0] * 8))
    assert em == 1 and not any(q)
