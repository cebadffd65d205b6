"""The Nx2D influence kernel where blocks of records are few (several warps share one)
and where steps bracket many receiver ranges (runs of eight at a depth), beside the
ordinary case, against eigenray runs, whose gather takes every record and receiver by
itself: as many contributions as hits, and no field at a receiver without one. Ranges
per step sit on both sides of 16, and no multiple of eight."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile3d import env_text, write_files

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nalpha,nrr,nrz", [(3, 1, 1), (1, 2003, 41), (3, 1601, 33), (3, 1609, 33), (5, 30, 301), (201, 61, 7)])
@pytest.mark.parametrize("beam", "BG")
def test_contributions(beam, nalpha, nrr, nrz, tmp_path):
    def env(run):
        return env_text(title="dense", freq=120.0, ssp_opt="CVW", depth=1000.0,
                        ssp=[(0.0, 1500.0), (400.0, 1490.0), (1000.0, 1510.0)], bot=("A", 1650.0, 1.6, 0.5), sx=[0.0],
                        sy=[0.0], sz=[250.0], rz=[300.0], rr_km=[4.0], theta=[0.0, 90.0],
                        run_type=run + beam + "   2", alpha=(nalpha, -25.0, 25.0) if nalpha > 1 else (1, 3.0, 3.0),
                        beta=(9, 0.0, 360.0), step=100.0, box_km=(10.2, 10.2), box_z=1100.0,
                        nrz_range=(nrz, 1.0, 999.0) if nrz > 1 else None, rr_range=(nrr, 0.0, 10.0) if nrr > 1 else None)
    root = os.path.join(str(tmp_path), "e")
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup3d(write_files({".env": env("C")}, root)).run()
        field, evals = t.field3d()[:, 0, 0], t.stats()["evals"]
    with B.Tracer(precision=B.PREC_FP64) as t:
        hits = t.setup3d(write_files({".env": env("E")}, root)).run().eigen_hits()
    assert evals == len(hits) and (evals > 0 or nalpha == 1 or nrr == 1)
    at = np.zeros(field.shape, bool)
    at[hits["isz"], hits["itheta"], hits["iz"], hits["ir"]] = True
    assert not np.any((field != 0) & ~at)


def test_more_items_than_a_pass(tmp_path):
    """15 ranges a step at 2.4 million depths: more than 2^25 items of a record, which take
    two passes. Depths are exact in FP32, so the two halves of the grid, one pass each,
    hold the same receivers: their contributions sum to the whole grid's."""
    def evals(i0, n):
        text = env_text(title="deep", freq=120.0, ssp_opt="CVW", depth=1000.0, ssp=[(0.0, 1500.0), (1000.0, 1510.0)],
                        bot=("A", 1650.0, 1.6, 0.5), sx=[0.0], sy=[0.0], sz=[250.0], rz=None, rr_km=None, theta=[0.0],
                        run_type="CB   2", alpha=(2, -3.0, 4.0), beta=(9, 0.0, 360.0), step=5000.0, box_km=(10.2, 10.2),
                        box_z=1100.0, nrz_range=(n, 256.0 + i0 / 8192.0, 256.0 + (i0 + n - 1) / 8192.0),
                        rr_range=(31, 0.0, 10.0))
        text = text.replace("%g %g /" % (256.0 + i0 / 8192.0, 256.0 + (i0 + n - 1) / 8192.0),
                            "%.13f %.13f /" % (256.0 + i0 / 8192.0, 256.0 + (i0 + n - 1) / 8192.0))
        with B.Tracer(precision=B.PREC_FP64) as t:
            t.setup3d(write_files({".env": text}, os.path.join(str(tmp_path), "e"))).run()
            return t.stats()["evals"]
    half = 1 << 20
    n = 2400000
    total = evals(0, n)
    assert total == evals(0, half) + evals(half, half) + evals(2 * half, n - 2 * half) > 15 * half
