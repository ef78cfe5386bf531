"""The single-CTA form of the beam's Newton kernel with an odd number of nodes (n + 16 floats of row
exponents, two more than a multiple of four, precede the matrices that it reads in 16-byte pieces),
against the oracle within the FP64 form's 1e-10."""
import pytest

from conftest import rel, seeded_vorticity
from fsibe_2d_gb300 import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [9, 13, 33, 64, 101, 301])
def test_single_cta_form_matches_the_oracle(oracle, monkeypatch, ns):
    import fsibe_2d_gb300 as F
    p = make_params(nx=64, ny=64, ns=ns, dt=1e-3)
    monkeypatch.setenv("FSIBE_BEAM_CLUSTER", "0")
    g = F.Run(p)
    monkeypatch.delenv("FSIBE_BEAM_CLUSTER")
    assert g.beam_cluster() == 0
    o = oracle.OracleRun(make_params(nx=64, ny=64, ns=ns, dt=1e-3))
    w = seeded_vorticity(64, seed=ns)
    g.init_fields(w)
    o.init_fields(w)
    g.time_step(12)
    o.time_step(12)
    assert g.scalars().status == 0
    assert rel(g.beam()[0][:2], o.beam()[0][:2]) < 1e-10 and rel(g.vort(), o.vort()) < 1e-10
    g.close()
    o.close()
