"""Beams whose spreading is not a finite number: a receiver test that compares with
NaN or infinity keeps the receiver, and so must every rule that leaves out work.

Against eigenray runs where they take every record and receiver by itself (beams in
ray-centred coordinates): as many contributions as hits."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env

pytestmark = pytest.mark.gpu


def run(s, root):
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup(write_env(s, root)).run()
        return (t.eigen_hits() if s.run_type[0] == "E" else t.field()), t.stats()


@pytest.mark.parametrize("beam", "gb")
def test_raycen_beam_shift_without_loss(beam, tmp_path):
    """The displacement of a beam at total reflection off a lossless bottom has NaN q."""
    s = EnvSpec(title="nan", freq=400.0, ssp_type="C", top_bc="R", atten_unit="W", ssp_z=np.linspace(0.0, 120.0, 6),
                ssp_cp=np.array([1509.3, 1504.7, 1496.0, 1497.3, 1499.3, 1506.7]), bot_bc="A",
                bot_hs=(120.0, 1600.0, 0.0, 1.7, 0.0, 0.0), nsz=1, sz=(24.0,), nrz=16, rz=(12.0, 114.0), nrr=31,
                rr_km=(-0.24, 1.2), run_type="C%s RR S" % beam, nalpha=2, alpha=(-20.0, 20.0), deltas=0.0, box_z=132.0,
                box_r_km=1.212)
    root = os.path.join(str(tmp_path), "e")
    field, st = run(s, root)
    s.run_type = "E%s RR S" % beam
    hits, _ = run(s, root)
    assert st["evals"] == len(hits) > 0
    assert np.isnan(field).any()
