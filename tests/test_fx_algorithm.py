"""The FP64 form's fixed-point transforms (fft_fx.cuh) restated on the CPU in exact integers.

The restatement follows the kernel's arithmetic bit for bit: rows of doubles on one exponent (59
bits for the largest component, 60 before the merge of a half spectrum), 62-bit twiddles in
balanced halves without the low x low products, the shifts that the growth and the sum of moduli
ask for, rounded to nearest.  It checks that no intermediate value leaves 64 bits, nor a twiddled
one 2^63, for the rows that stretch the bounds (constant, alternating, one spike, one mode at the
corner of the complex square, wide ranges), and that the error stays below that of FP64: each
transform's result within 2^-53 of its 2-norm, where the reference is a DFT of the same doubles
in extended precision."""
import math

import numpy as np
import pytest

LIM = 62
PI = math.pi


def dft_ld(z, sign):
    """DFT in long double by the definition's matrix (twiddles from long double cos and sin)."""
    n = len(z)
    k = np.arange(n)
    a = (np.outer(k, k) % n).astype(np.longdouble) * (sign * 2 * np.longdouble(np.pi)) / n
    # the constant pi to long double accuracy
    a = a * (np.longdouble("3.14159265358979323846264338327950288") / np.longdouble(np.pi))
    c, s = np.cos(a), np.sin(a)
    return c @ z.real - s @ z.imag, c @ z.imag + s @ z.real


def halves(v):
    lo = ((v + 2**31) % 2**32) - 2**31
    if lo == -2**31:
        v += 1
        lo += 1
    return (v - lo) >> 32, lo


def twiddle(m, n):
    one = np.longdouble(2) ** 62
    a = np.longdouble(2) * np.longdouble("3.14159265358979323846264338327950288") * m / n
    return halves(int(np.rint(np.cos(a) * one))) + halves(int(np.rint(-np.sin(a) * one)))


def split(a):
    lo = ((a + 2**31) % 2**32) - 2**31
    return (a - lo) >> 32, lo


def s64(v):
    assert -2**63 <= v < 2**63, "left 64 bits"
    return v


def cmul(a, w):
    (xh, xl), (yh, yl) = split(a[0]), split(a[1])
    ch, cl, sh, sl = w
    cr = s64(xh * cl + xl * ch - yh * sl - yl * sh + 2**29)
    ci = s64(xh * sl + xl * sh + yh * cl + yl * ch + 2**29)
    hr, hi = xh * ch - yh * sh, xh * sh + yh * ch
    return (s64((hr * 2**32 + cr) >> 30), s64((hi * 2**32 + ci) >> 30))


def mulh(a):
    HH, HL = 759250125, -25716447
    h, l = split(s64(a))
    return s64((h * HH * 2**32 + s64(h * HL + l * HH + 2**29)) >> 30)


def shr(a, s):
    return (a + (1 << s >> 1) + (a >> 63)) >> s if s else a


def dft8(v, inv):
    add = lambda a, b: (s64(a[0] + b[0]), s64(a[1] + b[1]))
    sub = lambda a, b: (s64(a[0] - b[0]), s64(a[1] - b[1]))
    rot = lambda a: (-a[1], a[0]) if inv else (a[1], -a[0])

    def dft4(x):
        a, b = add(x[0], x[2]), sub(x[0], x[2])
        c, d = add(x[1], x[3]), rot(sub(x[1], x[3]))
        return [add(a, c), add(b, d), sub(a, c), sub(b, d)]
    if len(v) == 2:
        return [add(v[0], v[1]), sub(v[0], v[1])]
    if len(v) == 4:
        return dft4(v)
    e = [add(v[i], v[i + 4]) for i in range(4)]
    t = [sub(v[i], v[i + 4]) for i in range(4)]
    o = [t[0], None, rot(t[2]), None]
    if not inv:
        o[1] = (mulh(t[1][0] + t[1][1]), mulh(t[1][1] - t[1][0]))
        o[3] = (mulh(t[3][1] - t[3][0]), -mulh(t[3][0] + t[3][1]))
    else:
        o[1] = (mulh(t[1][0] - t[1][1]), mulh(t[1][0] + t[1][1]))
        o[3] = (-mulh(t[3][0] + t[3][1]), mulh(t[3][0] - t[3][1]))
    e, o = dft4(e), dft4(o)
    return [e[0], o[0], e[1], o[1], e[2], o[2], e[3], o[3]]


def down(b0, g, lb):
    return max(min(b0 + g, lb) - LIM, 0)


def stages(z, inv, b0, late, lsum):
    """fx_stages: Stockham passes (radix 8, the last 4 or 2); returns (values, total shift)."""
    n = len(z)
    lb, ns, g, done = 44 + lsum.bit_length(), 1, 0, 0
    while ns < n:
        p = min(8, n // ns)
        g += p.bit_length() - 1
        d = 0 if (late and ns == 1) else down(b0, g, lb)
        z = [(shr(a, d - done), shr(b, d - done)) for a, b in z]
        done = d
        out = [None] * n
        for j in range(n // p):
            k = j & (ns - 1)
            v = [z[j + r * (n // p)] for r in range(p)]
            if ns > 1:
                w = [twiddle(r * k * (n // p) // ns, n) for r in range(p)]
                if inv:
                    w = [(a, b, -c, -e) for a, b, c, e in w]
                v = [v[0]] + [cmul(v[r], w[r]) for r in range(1, p)]
            v = dft8(v, inv)
            for r in range(p):
                out[(j - k) * p + k + r * ns] = v[r]
        z, ns = out, ns * p
    return z, done


def enter(x, bits):
    """Doubles on the scale of the largest: (integers, exponent)."""
    em = max(max(math.frexp(abs(v))[1] for v in x if v != 0.0), -900) if np.any(x != 0.0) else 0
    e = em - bits
    q = []
    for v in x:
        m, ex = math.frexp(v)
        m = int(math.ldexp(abs(m), 53))
        s = em - ex
        r = (((m << (bits - 53 + 1)) >> min(s, 63)) + 1) >> 1 if m else 0
        q.append(r if v >= 0 else -r)
    return q, e


l1 = lambda a: abs(a >> 44) + 1


def rows(n, seed):
    rng = np.random.default_rng(seed)
    k = np.arange(n)
    one = np.nextafter(1.0, 0.0)
    z = {"constant": np.full(n, one + 1j * one), "alternating": one * (1 - 2.0 * (k & 1)) * (1 + 1j),
         "spike": np.where(k == n // 3, (one + 1j * one), 0),
         "mode": one * np.sign(np.cos(2 * PI * 3 * k / n) + 1e-9) + 1j * one * np.sign(np.sin(2 * PI * 3 * k / n) + 1e-9),
         "noise": rng.standard_normal(n) + 1j * rng.standard_normal(n),
         "decaying": np.exp(-0.2 * k) * (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 1e-200,
         "wide": (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * 10.0 ** rng.uniform(-18, 3, n)}
    return z


@pytest.mark.parametrize("n", [16, 32, 64, 128, 512])
@pytest.mark.parametrize("inv", [False, True])
def test_complex_rows(n, inv):
    for name, z in rows(n, n).items():
        q, e = enter(np.concatenate([z.real, z.imag]), 59)
        v = list(zip(q[:n], q[n:]))
        out, d = stages(v, inv, 59, True, sum(l1(a) for a in q))
        # the kernel's last rounding is to double; here the integers themselves, less exact than
        # that by nothing the bound has not room for
        sc = np.longdouble(2) ** (e + d)
        re, im = dft_ld(z.astype(np.clongdouble), 1 if inv else -1)
        gr = np.array([np.longdouble(a) * sc for a, _ in out])
        gi = np.array([np.longdouble(b) * sc for _, b in out])
        err = np.sqrt(((gr - re) ** 2 + (gi - im) ** 2).sum() / (re**2 + im**2).sum())
        assert err < 2.0**-53, (name, float(err))
        assert max(max(abs(a), abs(b)) for a, b in out) < 2**63, name


@pytest.mark.parametrize("h", [16, 64, 256])
def test_half_spectrum_rows(h):
    """The merge of a half spectrum (60 bits) and its inverse transform stay in range and exact."""
    for name, z in rows(h, h + 1).items():
        x = z.copy()
        x[0] = x[0].real
        q, e = enter(np.concatenate([x.real, x.imag]), 60)
        X = list(zip(q[:h], q[h:]))
        Z = [None] * h
        for k in range(1, h // 2):
            a, c = X[k], X[h - k]
            s, d = (a[0] + c[0], a[1] - c[1]), (a[0] - c[0], a[1] + c[1])
            ch, cl, sh, sl = twiddle(k, 2 * h)
            o = cmul(d, (ch, cl, -sh, -sl))
            Z[k] = (s64(s[0] - o[1]), s64(s[1] + o[0]))
            Z[h - k] = (s64(s[0] + o[1]), s64(o[0] - s[1]))
        Z[0] = (X[0][0], X[0][0])
        Z[h // 2] = (2 * X[h // 2][0], -2 * X[h // 2][1])
        lsum = 3 * sum(l1(a) for a in q)
        assert sum(math.hypot(a, b) for a, b in Z) <= lsum * 2.0**44
        out, d = stages(Z, True, 62, False, lsum)
        sc = np.longdouble(2) ** (e + d)
        got = np.empty(2 * h, dtype=np.longdouble)
        got[0::2] = [np.longdouble(a) * sc for a, _ in out]
        got[1::2] = [np.longdouble(b) * sc for _, b in out]
        full = np.zeros(2 * h, dtype=np.clongdouble)
        full[:h] = x
        full[h + 1:] = np.conj(x[1:][::-1])
        re, im = dft_ld(full, 1)
        err = np.sqrt(((got - re) ** 2).sum() / (re**2).sum())
        assert err < 2.0**-53, (name, float(err))


@pytest.mark.parametrize("h", [16, 64, 256])
def test_real_rows_split(h):
    """The split of a forward transform's halves into the half spectrum stays in range and exact."""
    for name, z in rows(h, h + 2).items():
        q, e = enter(np.concatenate([z.real, z.imag]), 59)
        out, d = stages(list(zip(q[:h], q[h:])), False, 59, True, sum(l1(a) for a in q))
        hv = [(shr(a, 1), shr(b, 1)) for a, b in out]
        X = [None] * h
        for k in range(1, h // 2):
            a, c = hv[k], hv[h - k]
            s, dd = (s64(a[0] + c[0]), s64(a[1] - c[1])), (s64(a[1] + c[1]), s64(c[0] - a[0]))
            o = cmul(dd, twiddle(k, 2 * h))
            X[k] = (s64(s[0] + o[0]), s64(s[1] + o[1]))
            X[h - k] = (s64(s[0] - o[0]), s64(o[1] - s[1]))
        X[0] = (s64(2 * (hv[0][0] + hv[0][1])), 0)
        X[h // 2] = (2 * hv[h // 2][0], -2 * hv[h // 2][1])
        sc = np.longdouble(2) ** (e + d)
        x = np.empty(2 * h, dtype=np.clongdouble)
        x[0::2], x[1::2] = z.real, z.imag
        re, im = dft_ld(x, -1)
        gr = np.array([np.longdouble(a) * sc for a, _ in X])
        gi = np.array([np.longdouble(b) * sc for _, b in X])
        gi[0] = im[0]
        err = np.sqrt(((gr - re[:h]) ** 2 + (gi - im[:h]) ** 2).sum() / (re[:h]**2 + im[:h]**2).sum())
        # X[0] is a sum of two halves, each rounded at the last bit
        assert err < 2.0**-53, (name, float(err))
