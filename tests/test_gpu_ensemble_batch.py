"""Runs of one shape in one launch (the batches of an ensemble of 8 or more runs) against the runs alone:
batches of two and more, one run above a batch's capacity (16), oblong grids, odd node counts, both
precision forms, shapes without a batched form beside them, and a run that stops with an error beside
others that go on.  The kernels' batched forms are the same source; which multiply-add pairs are fused
is the compiler's, so FP64 states agree to refinement rounding (1e-12 of their 2-norm, the bound between
the forms of the beam kernel) and FP32-compensated ones within 1e-5."""
import numpy as np
import pytest

from conftest import rel, seeded_vorticity
from fsibe_2d_gb300 import make_params, FSIBE_FP32C, FSIBE_FP64

pytestmark = pytest.mark.gpu


def _p(nx, ny, ns, precision, k, **more):
    yl = 4.0 * ny / nx
    return make_params(nx=nx, ny=ny, ns=ns, yl=yl, x0=1.0, y0=0.5 * yl, precision=precision, dt=2e-4,
                       Re=100.0 + 37.0 * k, EI=0.05 + 0.02 * k, mu=1.0 + 0.1 * k, **more)


def _compare(r, p, w, steps):
    import fsibe_2d_gb300 as F
    alone = F.Run(p)
    alone.init_fields(w)
    for _ in range(steps):
        alone.step()
    tol = 1e-12 if p.precision == FSIBE_FP64 else 1e-5
    assert r.scalars().status == 0 and r.scalars().time == alone.scalars().time
    assert rel(r.vortk(), alone.vortk()) < tol and rel(r.u(), alone.u()) < tol
    assert rel(r.beam()[0][:2], alone.beam()[0][:2]) < tol
    assert rel(r.beam()[0][4], alone.beam()[0][4]) < max(tol, 1e-10)
    alone.close()


CASES = {
    "small": [(64, 64, 16, FSIBE_FP32C, 2), (128, 64, 17, FSIBE_FP64, 3), (64, 128, 9, FSIBE_FP32C, 2)],
    "above": [(64, 64, 16, FSIBE_FP32C, 17), (64, 64, 16, FSIBE_FP64, 1)],
    "large": [(1024, 512, 145, FSIBE_FP32C, 3), (512, 512, 128, FSIBE_FP64, 2), (2048, 256, 64, FSIBE_FP32C, 2)],
    "singles": [(256, 256, 64, FSIBE_FP32C, 42)],      # more beams than clusters are kept for
}


@pytest.mark.parametrize("name", list(CASES))
def test_batched_runs_match_their_single_runs(name):
    import fsibe_2d_gb300 as F
    ps = [_p(nx, ny, ns, prec, k) for nx, ny, ns, prec, n in CASES[name] for k in range(n)]
    ps.append(_p(128, 128, 32, FSIBE_FP32C, 1, iSponge=1, SpongeSize=0.5, eps_sponge=1e-2))
    ens = F.Ensemble(ps)
    assert (ens.runs[0].beam_cluster() == 0) == (name == "singles")
    ws = [seeded_vorticity(p.nx, ny=p.ny, seed=k) for k, p in enumerate(ps)]
    for r, w in zip(ens.runs, ws):
        r.init_fields(w)
    ens.step(9)
    for p, w, r in list(zip(ps, ws, ens.runs))[-20:]:
        _compare(r, p, w, 9)
    ens.close()


def test_a_stopped_run_leaves_its_batch_alone():
    import fsibe_2d_gb300 as F
    ps = [_p(64, 64, 16, FSIBE_FP64, k) for k in range(8)]
    ps[1].newton_maxit = 1
    ens = F.Ensemble(ps)
    ws = [seeded_vorticity(64, seed=k) for k in range(8)]
    for r, w in zip(ens.runs, ws):
        r.init_fields(w)
    with pytest.raises(F.FsibeError):
        ens.step(6)
    assert ens.runs[1].scalars().status == 4        # FSIBE_ERR_NEWTON_MAXIT
    for k in (0, 2, 7):
        _compare(ens.runs[k], ps[k], ws[k], 6)
    ens.close()
