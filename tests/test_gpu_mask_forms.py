"""The FP64 raster (k_mask_raster_d) where its choice of the winner by distance can go wrong: beams so
thick that SmoothStep is exactly 1 over many cells (ties: the first drawn wins), a sharp mask (every
value 0 or 1), a straight beam (equal distances to neighbouring segments), a bent one, the sharp
trailing end, and walls or a cylinder as background, redrawn as the beam moves.  Against the oracle: the
mask and the products of the mask and its velocity, which are what the equations use, to 1e-13 of the
largest mask.  (Where SmoothStep is within a rounding of zero, which primitive's velocity a cell carries
depends on the last bit of erf.)"""
import numpy as np
import pytest

from conftest import seeded_vorticity
from fsibe_2d_gb300 import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(), dict(thickness_cells=24.0), dict(N_smooth=0.0), dict(iSharpTrailing=1), dict(angle_beam=17.0),
    dict(iWalls=1, h_channel=0.3), dict(iCylinder=1, R_cylinder=0.1), dict(iSponge=4, SpongeSize=0.5),
    dict(iWalls=1, h_channel=0.3, thickness_cells=16.0, iCylinder=1, R_cylinder=0.2)], ids=str)
def test_fp64_mask_of_a_moving_beam(oracle, kw):
    import fsibe_2d_gb300 as F
    n = 128
    p = make_params(nx=n, ny=n, ns=33, dt=1e-3, **kw)
    g, o = F.Run(p), oracle.OracleRun(p)
    w = seeded_vorticity(n, seed=9)
    g.init_fields(w); o.init_fields(w)
    s = np.linspace(0.0, 1.0, 33)
    zero = np.zeros(33)
    for amp in (0.0, 0.05, -0.2):   # straight, then bent one way and the other: the box moves
        a = np.deg2rad(kw.get("angle_beam", 0.0))
        y = amp * s**2
        x = s - 0.5 * amp**2 * s**3
        bx, by = 1.0 + x * np.cos(a) - y * np.sin(a), 2.0 + x * np.sin(a) + y * np.cos(a)
        b = np.stack([bx, by, 0.3 * s, np.sin(3 * s), 2 * amp * s, zero])
        for r in (g, o):
            r.set_beam(b, zero, zero, zero, zero)
            r.create_mask(0.0)
        mg, mo = g.mask(), o.mask()
        for q in range(3):
            fg, fo = (m[0] if q == 0 else m[0] * m[q] for m in (mg, mo))
            assert np.abs(fg - fo).max() <= 1e-13 * np.abs(mo[0]).max(), (kw, amp, q, np.abs(fg - fo).max())
    g.close(); o.close()
