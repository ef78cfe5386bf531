"""The FP64 form's fixed-point transforms on the GPU (fft_fx.cuh) through coftxy and cofitxy.

Every transform length and stage structure (radix 8 with a last 8, 4 or 2; rows within a warp and
over several), on the row shapes that stretch a common exponent: a spike, a thin layer over noise,
rows and elements of widely different size.  The reference is numpy's transform in extended
precision.  Tolerance: each of the two passes rounds its results to double (2^-53 of each element
at most) and the fixed-point part is below 2^-54 of the row's 2-norm a pass, so the sum stays below
3 2^-53 of the 2-norm; an FP64 transform of these sizes is at 2 to 3 10^-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L, TOL = np.longdouble, 3.0 * 2.0**-53


def _packed(f):
    ny, nx = f.shape
    h = nx // 2
    ft = np.fft.fft(np.fft.rfft(f.astype(L), axis=1)[:, :h], axis=0) / L(nx * ny)
    out = np.zeros((ny, nx), dtype=L)
    out[0, 0::2], out[0, 1::2] = ft[0].real, ft[0].imag
    j = np.arange(1, ny // 2)
    p, m = ft[j], ft[ny - j]
    out[2 * j, 0::2], out[2 * j + 1, 0::2] = (p.real + m.real) / 2, (p.imag - m.imag) / 2
    out[2 * j, 1::2], out[2 * j + 1, 1::2] = (p.imag + m.imag) / 2, (m.real - p.real) / 2
    return out


def _physical(pk):
    ny, nx = pk.shape
    h = nx // 2
    pk = pk.astype(L)
    ft = np.zeros((ny, h + 1), dtype=np.clongdouble)
    ft[0, :h] = pk[0, 0::2] + 1j * pk[0, 1::2]
    j = np.arange(1, ny // 2)
    a, b, c, d = pk[2 * j, 0::2], pk[2 * j + 1, 0::2], pk[2 * j, 1::2], pk[2 * j + 1, 1::2]
    ft[j, :h] = (a - d) + 1j * (b + c)
    ft[ny - j, :h] = (a + d) + 1j * (c - b)
    g = np.fft.ifft(ft, axis=0) * ny
    g[:, 0] = g[:, 0].real
    return np.fft.irfft(g, n=nx, axis=1) * nx


def _fields(nx, ny):
    rng = np.random.default_rng(nx + 3 * ny)
    x, y = np.arange(nx) / nx, np.arange(ny)[:, None] / ny
    spike = np.zeros((ny, nx))
    spike[3, 5] = 1.0 / 3.0
    noise = rng.standard_normal((ny, nx))
    return {"noise": noise, "smooth": np.exp(np.cos(2 * np.pi * x)) * np.exp(np.sin(2 * np.pi * y)), "spike": spike,
            "layer": np.where(np.abs(y - 0.5) * ny < 3, 1e4, 0.0) * np.exp(-((x - 0.4) * 8) ** 2) + 1e-6 * noise,
            "rows": noise * 10.0 ** rng.uniform(-12, 12, (ny, 1)), "tiny": noise * 1e-250,
            "elements": noise * 10.0 ** rng.uniform(-12, 0, (ny, nx))}


def _rel(a, b):
    s = np.abs(b).max()
    a, b = a / s, b / s
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("nx,ny", [(32, 32), (64, 128), (128, 64), (256, 512), (1024, 256), (2048, 64), (64, 2048),
                                   (32, 4096)])
def test_transforms_within_fp64(nx, ny):
    import fsibe_2d_gb300 as F
    r = F.Run(F.make_params(nx=nx, ny=ny, ns=16, precision=F.FSIBE_FP64))
    for name, f in _fields(nx, ny).items():
        fk = r.coftxy(f)
        assert _rel(fk, _packed(f)) < TOL, (name, "forward")
        assert _rel(r.cofitxy(fk), _physical(fk)) < TOL, (name, "inverse")
    r.close()


def test_zero_and_non_finite_rows():
    import fsibe_2d_gb300 as F
    r = F.Run(F.make_params(nx=256, ny=64, ns=16, precision=F.FSIBE_FP64))
    assert not r.coftxy(np.zeros((64, 256))).any()
    for bad in (np.nan, np.inf, -np.inf):
        f = np.ones((64, 256))
        f[17, 200] = bad
        assert np.isnan(r.coftxy(f)).any()
    r.close()
