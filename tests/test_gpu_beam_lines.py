"""The beam kernel on both sides of its lines: 8 and 16 CTAs (144 nodes), the boundary equations' own CTAs
and M^-1 in shared memory (298, 318 nodes), the position sums by the serial loop and by events (544).
The cluster form against the single-CTA form, and 16 CTAs against 8 where both run: they agree to
refinement rounding (1e-12 of the 2-norm, the bound between the forms), and the positions' sums are the
serial loop's in each."""
import pytest

from conftest import rel, seeded_vorticity
from fsibe_2d_gb300 import make_params

pytestmark = pytest.mark.gpu


def _run(monkeypatch, ns, cluster):
    import fsibe_2d_gb300 as F
    n = 256 if ns <= 256 else 512
    if cluster is not None:
        monkeypatch.setenv("FSIBE_BEAM_CLUSTER", str(cluster))
    r = F.Run(make_params(nx=n, ny=n, ns=ns, Re=300.0, dt=5e-5))
    monkeypatch.delenv("FSIBE_BEAM_CLUSTER", raising=False)
    r.init_fields(seeded_vorticity(n, seed=ns))
    r.time_step(10)
    assert r.scalars().status == 0
    return r


@pytest.mark.parametrize("ns,ctas", [(144, 8), (145, 16), (297, 16), (298, 16), (299, 16), (302, 16), (305, 16), (318, 16),
                                     (319, 16), (320, 16), (321, 16), (543, 16), (544, 16), (545, 16), (546, 16)])
def test_forms_agree_on_both_sides(monkeypatch, ns, ctas):
    a, s = _run(monkeypatch, ns, None), _run(monkeypatch, ns, 0)
    assert a.beam_cluster() == ctas and s.beam_cluster() == 0
    others = [_run(monkeypatch, ns, 8)] if ctas == 16 else []
    for o in [s] + others:
        assert rel(a.beam()[0], o.beam()[0]) < 1e-12
        assert a.scalars().newton_iters == o.scalars().newton_iters
        o.close()
    a.close()
