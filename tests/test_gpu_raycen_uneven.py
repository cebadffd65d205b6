"""Ray-centred geometric beams at receivers whose ranges are no even grid. The index
of a range (RToIR) takes the last spacing for all of them, so a record's two ends
say nothing of where the receivers between its indices lie, and no record may be
left out by its ends.

Against eigenray runs, whose gather takes every record and depth by itself: as many
contributions as hits, and no field at a receiver without one."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env
from bellhopcuda_b200.workloads import munk_c

pytestmark = pytest.mark.gpu

RANGES = {
    "squares": tuple(15.0 * np.linspace(0.05, 1.0, 41) ** 2),
    "last_spacing_small": tuple(np.linspace(0.0, 14.0, 40)) + (14.001,),
    "last_spacing_large": tuple(np.linspace(0.1, 5.0, 20)) + (15.0,),
    "one_moved": tuple(np.delete(np.linspace(0.0, 15.0, 41), 17)),
    "from_behind": (-3.0, -2.9, -0.5, 0.0, 1.0, 1.5, 7.0, 9.5, 10.0),
}


@pytest.mark.parametrize("beam", "bg")
@pytest.mark.parametrize("ranges", sorted(RANGES))
def test_uneven_ranges(ranges, beam, tmp_path):
    z = np.linspace(0.0, 1500.0, 31)
    rr = RANGES[ranges]
    s = EnvSpec(title="uneven", freq=120.0, ssp_type="C", top_bc="V", atten_unit="W", ssp_z=z, ssp_cp=munk_c(z * 3.0),
                bot_bc="A", bot_hs=(1500.0, 1650.0, 0.0, 1.7, 0.5, 0.0), nsz=2, sz=(430.0, 900.0), nrz=9,
                rz=(20.0, 1480.0), nrr=len(rr), rr_km=rr, run_type="C%s RR " % beam, nalpha=61, alpha=(-50.0, 50.0),
                deltas=0.0, box_z=1600.0, box_r_km=15.5)
    root = os.path.join(str(tmp_path), "e")
    with B.Tracer(precision=B.PREC_FP64) as t:
        field = t.setup(write_env(s, root)).run().field()
        st = t.stats()
    s.run_type = "E%s RR " % beam
    with B.Tracer(precision=B.PREC_FP64) as t:
        hits = t.setup(write_env(s, root)).run().eigen_hits()
    assert len(hits) > 0 and st["evals"] == len(hits)
    at = np.zeros(field.shape, bool)
    at[hits["isz"], hits["iz"], hits["ir"]] = True
    assert not np.any((field != 0) & ~at)
