"""The beam kernels' running sums by events (fsibe_2d_gb300/csrc/running_sum.cuh), restated in Python and
checked on the CPU against the serial FP64 loop, bit for bit.

Approximate sums in fixed point give every running value's binade where the error bound leaves no
doubt; steps within a binade are integer increments on its grid, formed without the running value; the
rest -- binade changes, ties, zeros, values near a power of two -- are events, FP64 additions walked in
order.  The restatement must give the serial loop's bits on every row it does not leave to that loop."""
import math
import random

import pytest

from test_running_sum_algorithm import FRAC, T52, bits, from_bits, term_inc

RS_EVENTS = 96


def fix(a, em):
    b = bits(a)
    e = (b >> 52) & 0x7FF
    v = ((b & FRAC) | T52) >> min(em - e + 2, 63)
    return -v if b >> 63 else v


def advance(cur, d):
    if d == 0:
        return cur
    b = bits(cur)
    m = (b & FRAC) | T52
    m = (-m if b >> 63 else m) + d
    return from_bits((b & ~FRAC) | (abs(m) & FRAC))


def running_sum(a):
    """(sums or None, events)."""
    n = len(a)
    em = max((bits(x) >> 52) & 0x7FF for x in a)
    if em == 0x7FF or em < 64:
        return None, 0
    q = [fix(x, em) for x in a]
    err = 2 * n + (sum(abs(v) for v in q) >> 41)

    def binade(v):
        lo, hi = abs(v) - err, abs(v) + err
        if lo <= 0 or lo.bit_length() != hi.bit_length():
            return 0
        return -lo.bit_length() if v < 0 else lo.bit_length()
    pre, event, p, s, b = [], [], 0, 0, 0
    for k in range(n):
        s += q[k]
        assert abs(s) < 2**62
        nxt = binade(s)
        ok = tie = False
        inc = 0
        if b and b == nxt:
            inc, ok, tie = term_inc(a[k], abs(b) - 53 + em - 1073)
        pre.append(p)
        event.append(not ok or tie)
        if not event[-1]:
            p += inc
        b = nxt
    if sum(event) > RS_EVENTS:
        return None, sum(event)
    out, start, base = [0.0] * n, 0.0, 0
    for k in range(n):
        out[k] = advance(start, pre[k] - base) if k else 0.0
        if event[k]:
            start, base = out[k] + a[k], pre[k]
    return out, sum(event)


def serial(a):
    out, s = [], 0.0
    for x in a:
        out.append(s)
        s = s + x
    return out


def check(a):
    got, ev = running_sum(a)
    if got is None:
        return None
    assert [bits(x) for x in got] == [bits(x) for x in serial(a)]
    return ev


@pytest.mark.parametrize("n", [129, 256, 257, 513, 1024, 2048])
def test_beam_rows(n):
    rng = random.Random(n)
    taken = 0
    for amp in (1e-9, 1e-4, 0.3):
        ph = rng.uniform(0, 6)
        th = [amp * math.sin(3 * i / n + ph) * (i / n) ** 2 + 1e-3 * amp * rng.uniform(-1, 1) for i in range(n)]
        for row in ([math.cos(t) / n for t in th], [math.sin(t) / n for t in th],
                    [-(0.1 * math.sin(5 * i / n) * math.sin(t) / n) for i, t in enumerate(th)]):
            taken += check(row) is not None
    assert taken >= 6  # the rows the kernels meet do not end in the serial loop


def test_hard_rows():
    rng = random.Random(5)
    n = 600
    rows = {"ties": [1.0] + [2.0**-53] * 300 + [3 * 2.0**-53] * (n - 301),
            "cancel": [1.0, -1.0] * (n // 2), "huge": [1e300] * n, "subnormal": [5e-324] * n,
            "mixed": [rng.uniform(-1, 1) * 10.0 ** rng.uniform(-20, 2) for _ in range(n)],
            "zeros": [0.0, -0.0] * (n // 2), "powers": [2.0 ** -(i % 60) for i in range(n)],
            "grow": [1e-12 * 1.05**i for i in range(n)], "down": [1.0] + [-(2.0**-11)] * (n - 1),
            "walk": [rng.choice((-1, 1)) * rng.uniform(0.5, 1) for _ in range(n)],
            "inf": [1.0] * 300 + [math.inf] + [1.0] * 299}
    for name, row in rows.items():
        check(row)
