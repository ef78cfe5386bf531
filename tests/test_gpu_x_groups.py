"""The x pass with a group of threads a transform (k_nl_x_g, k_stress_x_g, k_press_x_g) and the place of
a row's elements in shared memory.

On the CPU: the FP32 form's place of an element is a permutation that keeps the exchanges' half warps
in sixteen different bank pairs.  On the GPU: grids of every length the group kernels take in the FP32
form and of the first above it, oblong both ways, with the sponges' variants, against the oracle.
Tolerances: 1e-5 (FP32-compensated) and 1e-10 (FP64) of the fields' 2-norm, as for every feature."""
import pytest

from conftest import rel, seeded_vorticity
from fsibe_2d_gb300 import make_params, FSIBE_FP32C


def _place(i):
    return i ^ (((i >> 4) & 7) | ((i >> 3) & 8))


@pytest.mark.parametrize("n", [16, 32, 64, 128, 512, 2048, 4096])
def test_places_are_a_permutation_without_bank_conflicts(n):
    assert sorted(_place(i) for i in range(n)) == list(range(n))
    for t0 in range(0, n // 8 - 15, 16):            # a half warp's lanes t0 .. t0 + 15 of n / 8
        for q in range(8):                          # loads t + q n/8, and stores 8 t + q of the first stage
            if n >= 128:
                assert len({_place(t + q * (n // 8)) % 16 for t in range(t0, t0 + 16)}) == 16
            assert len({_place(8 * t + q) % 16 for t in range(t0, t0 + 16)}) == 16


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(FSIBE_FP32C, 1e-5), (0, 1e-10)])
@pytest.mark.parametrize("nx,ny,more", [
    (32, 32, {}), (64, 32, {}), (128, 64, dict(iSponge=1, SpongeSize=0.3, eps_sponge=1e-2)), (256, 512, {}),
    (512, 256, dict(iSponge=2, SpongeSize=0.3, eps_sponge=1e-2)), (512, 512, dict(iSponge=10, SpongeSize=1.0, eps_sponge=0.1)),
    (1024, 512, {})])
def test_x_pass_matches_the_oracle(oracle, nx, ny, more, precision, tol):
    import fsibe_2d_gb300 as F
    xl, yl = 4.0, 4.0 * ny / nx
    kw = dict(nx=nx, ny=ny, ns=max(9, nx // 4), xl=xl, yl=yl, x0=1.0, y0=0.5 * yl, Re=200.0, dt=1e-4, **more)
    w = seeded_vorticity(nx, ny=ny, seed=nx + ny)
    g, o = F.Run(make_params(precision=precision, **kw)), oracle.OracleRun(make_params(**kw))
    g.init_fields(w)
    o.init_fields(w)
    rg, ro = g.time_step(12), o.time_step(12)
    err = {"vorticity": rel(g.vort(), o.vort()), "u": rel(g.u(), o.u()), "press": rel(g.press(), o.press()),
           "drag": rel(rg[:, 10], ro[:, 10])}
    assert max(err.values()) < tol, err
    g.close()
    o.close()
