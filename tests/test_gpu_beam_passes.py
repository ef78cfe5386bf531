"""The cluster form of the beam's Newton kernel where its row partition and its early decisions can go
wrong: odd and even ns at the edges of the cluster sizes and of the rule that leaves the boundary
equations alone in the first and last CTA, and stopping tolerances on both sides of what one Newton
iteration leaves.  The number of Newton iterations of every step is that of the single-CTA form, which
solves for 2^-30 of every update; positions, angles and rates match the oracle within the FP64 form's
1e-10."""
import numpy as np
import pytest

from conftest import rel, seeded_vorticity
from fsibe_2d_gb300 import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,cluster", [(9, 4), (13, 4), (14, 8), (15, 8), (16, 8), (17, 8), (64, 8), (143, 8), (145, 16),
                                        (256, 16), (317, 16), (319, 16), (601, 16)])
@pytest.mark.parametrize("tol,EI", [(1e-10, 0.1), (1e-14, 0.01)])
def test_iterations_and_state(oracle, monkeypatch, ns, cluster, tol, EI):
    import fsibe_2d_gb300 as F
    kw = dict(nx=64, ny=64, ns=ns, dt=2e-4, newton_tol=tol, EI=EI)
    w = seeded_vorticity(64, seed=ns, sigma=0.05)
    g, o = F.Run(make_params(**kw)), oracle.OracleRun(make_params(**kw))
    monkeypatch.setenv("FSIBE_BEAM_CLUSTER", "0")
    s = F.Run(make_params(**kw))
    monkeypatch.delenv("FSIBE_BEAM_CLUSTER")
    assert g.beam_cluster() == cluster and s.beam_cluster() == 0
    for r in (g, o, s):
        r.init_fields(w)
    for _ in range(12):
        for r in (g, o, s):
            r.step()
        assert g.scalars().status == 0 and g.scalars().newton_iters == s.scalars().newton_iters
    gb, ob = g.beam()[0], o.beam()[0]
    for q in range(6):
        assert rel(gb[q], ob[q]) < 1e-10 or np.abs(gb[q] - ob[q]).max() < 1e-15, q
    for r in (g, o, s):
        r.close()
