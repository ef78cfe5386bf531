"""FP32 runs of a batch against the runs alone, element by element: a mistake confined to a few cells does
not show in a 2-norm.

The batched kernels are the same source, so the two differ by which multiply-add pairs the compiler fuses.
Tolerance, of a field's largest magnitude: a 2-D FP32 transform of 2^16 elements has 16 butterfly levels
of rounding, a standard deviation of about 2 units of 2^-24 of the rms, and the largest of 65536 such
differences between two results is below 16 units (2^-20); twice that for the velocity and the vorticity.
The pressure's right-hand side is a sum of larger terms that cancel: 2^-17."""
import numpy as np
import pytest

from conftest import seeded_vorticity
from fsibe_2d_gb300 import make_params, FSIBE_FP32C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ns", [(64, 64, 16), (256, 256, 64), (512, 128, 101), (1024, 64, 40)])
def test_batched_fields_element_by_element(nx, ny, ns):
    import fsibe_2d_gb300 as F
    yl = 4.0 * ny / nx
    ps = [make_params(nx=nx, ny=ny, ns=ns, yl=yl, x0=1.0, y0=0.5 * yl, precision=FSIBE_FP32C, dt=1e-4, Re=150.0 + 30 * k,
                      EI=0.05 + 0.01 * k) for k in range(9)]
    ws = [seeded_vorticity(nx, ny=ny, seed=10 + k) for k in range(9)]
    ens = F.Ensemble(ps)
    for r, w in zip(ens.runs, ws):
        r.init_fields(w)
    ens.step(4)
    for k in (0, 5, 8):
        alone = F.Run(ps[k])
        alone.init_fields(ws[k])
        for _ in range(4):
            alone.step()
        r = ens.runs[k]
        for name, tol in (("u", 2.0**-19), ("vort", 2.0**-19), ("press", 2.0**-17)):
            a, b = getattr(r, name)(), getattr(alone, name)()
            assert np.abs(a - b).max() <= tol * np.abs(b).max(), (k, name, np.abs(a - b).max() / np.abs(b).max())
        alone.close()
    ens.close()
