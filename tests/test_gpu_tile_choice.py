"""The x kernels' tiles are chosen for the steps that a context makes: k_press_x with the viscous stresses
inside (ensembles of 8 or more runs, FSIBE_STRESS_SPLIT=0) is another body than without them, and the
paired kernel has no such form, so that tile_config names it only where the steps launch it."""
import numpy as np
import pytest

from conftest import seeded_vorticity
from fsibe_2d_gb300 import make_params, FSIBE_FP32C

pytestmark = pytest.mark.gpu
PAIRED = 16                                             # the paired kernel's marker in tile_config


def _p(k=0, **more):
    return make_params(nx=128, ny=128, ns=32, precision=FSIBE_FP32C, Re=100.0 + k, dt=2e-4, **more)


@pytest.mark.parametrize("paired", [None, "1"])
def test_ensemble_tiles_are_those_of_its_own_steps(monkeypatch, paired):
    import fsibe_2d_gb300 as F
    if paired:
        monkeypatch.setenv("FSIBE_PX_PAIRED", paired)
    alone = F.Run(_p())                                 # tuned, and kept for the size, with the stresses apart
    assert not paired or alone.tile_config()[1][1] == PAIRED
    ens = F.Ensemble([_p(k) for k in range(8)])
    monkeypatch.setenv("FSIBE_STRESS_SPLIT", "0")
    inside = F.Run(_p())
    monkeypatch.delenv("FSIBE_STRESS_SPLIT")
    again = F.Run(_p())
    assert inside.tile_config()[1][1] != PAIRED
    assert all(r.tile_config() == inside.tile_config() for r in ens.runs)
    assert again.tile_config() == alone.tile_config()
    # what rounds differently is one choice for the size
    assert len({r.press_y_engine() for r in (alone, inside, again, *ens.runs)}) == 1
    inviscid = F.Run(_p(iViscous=0))                    # no stresses: the paired kernel may run
    assert not paired or inviscid.tile_config()[1][1] == PAIRED
    w = seeded_vorticity(128, seed=1)
    for r in ens.runs:
        r.init_fields(w)
    ens.step(3)
    assert all(r.scalars().status == 0 for r in ens.runs) and np.isfinite(ens.runs[7].vort()).all()
    for r in (alone, inside, again, inviscid):
        r.close()
    ens.close()
