"""The ends of the exponent range in the FP64 form's transforms, through coftxy and cofitxy: fields whose
values are near the largest double, below the smallest scale that the fixed-point rows take as it is
(2^-927), and denormal.  The reference is numpy's transform in extended precision.  Tolerance: that of the
ordinary scales (test_gpu_fx.py, 3 2^-53 of the 2-norm) and, for results below the normal range, two units
of the smallest denormal a pass in each element the pass sums."""
import numpy as np
import pytest

from test_gpu_fx import TOL, _packed, _physical

pytestmark = pytest.mark.gpu
L = np.longdouble


def _check(a, b, nsum, what):
    s = np.abs(b).max()
    norm = np.sqrt(((b / s) ** 2).sum()) * s
    err = np.sqrt((((a - b) / s) ** 2).sum()) * s
    assert np.isfinite(a).all(), what
    assert err <= TOL * norm + 2 * L(2.0) ** -1074 * np.sqrt(L(b.size)) * nsum, (what, float(err / norm))


@pytest.mark.parametrize("nx,ny", [(64, 128), (1024, 64), (32, 1024)])
@pytest.mark.parametrize("scale", [2.0**1006, 2.0**1003, 2.0**-925, 2.0**-930, 1e-300, 1e-307, 1e-312])
def test_fields_at_the_ends_of_the_range(nx, ny, scale):
    import fsibe_2d_gb300 as F
    r = F.Run(F.make_params(nx=nx, ny=ny, ns=16, precision=F.FSIBE_FP64))
    f = np.random.default_rng(nx).uniform(-1.0, 1.0, (ny, nx)) * scale
    f[ny // 2] = 0.0                                     # a row of zeros among them
    fk = r.coftxy(f)
    _check(fk, _packed(f), 1, "forward")                 # (the normalisation divides a pass's sums)
    g = f / (nx * ny) * 2.0**10 if scale > 1.0 else f    # a spectrum whose sums stay finite
    _check(r.cofitxy(g), _physical(g), nx + 1, "inverse")
    r.close()
